// dropin.cu -- the reference's hopping entry points on host arrays
// (include/dirac.h; reference lib/dirac.c:35-791).
//
// Each call copies the input parity of `qin` (API layout, host) to the
// device, converts it to the kernel layout, runs the sm_100a hopping kernel
// and copies the output parity back into `qout`; the other half of `qout` is
// not touched, as in the reference. The reference reads the links on every
// call, so by default so does this path: the link array is uploaded on
// every call, unless the caller has registered it with
// plqcd_gauge_update(u), which declares "these links are current until the
// next plqcd_gauge_update": then it is uploaded once and kept on the device.
// PLQCD_GAUGE_CACHE=1 keeps any link array by host address plus a
// fingerprint of sampled words (for callers known never to change links in
// place); PLQCD_GAUGE_CACHE=0 uploads on every call even when registered.
// The return value is the call's wall-clock seconds
// (lib/dirac.c:405-407), or -1 on failure with the reason in
// plqcd_last_error(). Calls are serialised (the reference is not
// re-entrant either: lib/dirac.c:12-13 and the global phip/phim buffers).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "dirac.h"
#include "internal.h"

using namespace plqcd;

namespace {

// t-slab chunks of the copy/compute pipeline (chunk_plan)
constexpr int kMaxChunks = 64;

// what a device copy of the links was loaded from. `dirty`: nothing, or an
// array declared changed since (plqcd_gauge_update marks every copy; only the
// copy's own upload clears the mark)
struct LinkCache {
    const void *u = nullptr;   // host array (split family: its real plane)
    const void *im = nullptr;  // split family: the imaginary plane
    int lanes = 0;             // lane-packed family
    uint64_t fp = 0;
    bool dirty = true;
};

// what a captured pipeline graph depends on besides the device buffers
struct GraphKey {
    const void *src = nullptr, *dst = nullptr;
    int parity = 0, plan = 0;  // plan: chunk_plan's id
    unsigned flags = 0;
    const void *gauge = nullptr;
    bool operator==(const GraphKey &o) const {
        return src == o.src && dst == o.dst && parity == o.parity && plan == o.plan && flags == o.flags &&
               gauge == o.gauge;
    }
};
constexpr int kGraphSlots = 4;

struct DropIn {
    plqcd_gauge *gauge_split = nullptr, *gauge12 = nullptr;
    LinkCache split18, split12;
    int dims[4] = {0, 0, 0, 0};
    cudaStream_t s_h2d = nullptr, s_d2h = nullptr;  // copy streams
    cudaEvent_t ev_in[kMaxChunks] = {}, ev_out[kMaxChunks] = {}, ev_k0[kMaxChunks] = {}, ev_k1[kMaxChunks] = {};
    plqcd_lattice *lat = nullptr;
    plqcd_gauge *gauge = nullptr;
    void *aos_in = nullptr, *aos_out = nullptr;  // API layout staging, one parity
    void *f_in = nullptr, *f_out = nullptr;      // kernel layout (F64), one parity
    LinkCache links;                             // of `gauge`
    cudaStream_t stream = nullptr;  // owned by the drop-in path
    double kernel_ms = 0, h2d = 0, d2h = 0;
    cudaEvent_t ev_fork = nullptr, ev_join[2] = {nullptr, nullptr};  // capture fork / join
    GraphKey graph_key[kGraphSlots];
    cudaGraphExec_t graph_exec[kGraphSlots] = {};
    int graph_next = 0;
    GraphKey last_key;
    bool last_valid = false;
    // lane-packed entry points (spinor_256 / spinor_512 and su3_256 / su3_512)
    plqcd_gauge *gauge_packed = nullptr, *gauge_packed12 = nullptr;
    LinkCache packed18, packed12;
};

std::mutex g_mu;
DropIn g_d;
// the link array declared current by plqcd_gauge_update. release_locked
// keeps it, so a registration made between init_plqcd and the first call
// survives that call's set-up (device copies still start out dirty);
// finalize_plqcd clears it.
const void *g_registered = nullptr;

void release_locked() {
    if (g_d.lat) cudaSetDevice(g_d.lat->device);
    if (g_d.gauge) plqcd_gauge_destroy(g_d.gauge);
    if (g_d.gauge_split) plqcd_gauge_destroy(g_d.gauge_split);
    if (g_d.gauge12) plqcd_gauge_destroy(g_d.gauge12);
    if (g_d.gauge_packed) plqcd_gauge_destroy(g_d.gauge_packed);
    if (g_d.gauge_packed12) plqcd_gauge_destroy(g_d.gauge_packed12);
    void *bufs[4] = {g_d.aos_in, g_d.aos_out, g_d.f_in, g_d.f_out};
    for (void *b : bufs)
        if (b) cudaFree(b);
    for (cudaGraphExec_t x : g_d.graph_exec)
        if (x) cudaGraphExecDestroy(x);
    for (int c = 0; c < kMaxChunks; c++)
        for (cudaEvent_t ev : {g_d.ev_in[c], g_d.ev_out[c], g_d.ev_k0[c], g_d.ev_k1[c]})
            if (ev) cudaEventDestroy(ev);
    for (cudaEvent_t ev : {g_d.ev_fork, g_d.ev_join[0], g_d.ev_join[1]})
        if (ev) cudaEventDestroy(ev);
    if (g_d.s_h2d) cudaStreamDestroy(g_d.s_h2d);
    if (g_d.s_d2h) cudaStreamDestroy(g_d.s_d2h);
    if (g_d.lat) plqcd_lattice_destroy(g_d.lat);
    if (g_d.stream) cudaStreamDestroy(g_d.stream);
    g_d = DropIn();
}

bool env_flag(const char *name, bool dflt) {
    const char *v = getenv(name);
    if (!v || !*v) return dflt;
    return !(v[0] == '0' || v[0] == 'n' || v[0] == 'N' || v[0] == 'f' || v[0] == 'F');
}

int env_int_dropin(const char *name, int dflt) {
    const char *v = getenv(name);
    return (v && *v) ? atoi(v) : dflt;
}

// Chunk boundaries in t-slabs, bound[0] = 0 ... bound[nch] = L3. Default:
// chunk sizes 1, 1, 2, 4, ... up to `cap` slabs, from both ends inward, so
// the chunks that cross PCIe alone (the first three up, the last two or
// three down) are one slab each and the middle ones are large.
// PLQCD_DROPIN_CHUNKS=n: n equal chunks instead; PLQCD_DROPIN_CAP: the cap
// (default L3/8).
int chunk_plan(int L3, int *bound, int *plan_id) {
    const int uniform = env_int_dropin("PLQCD_DROPIN_CHUNKS", 0);
    if (uniform > 0) {
        const int n = uniform > kMaxChunks ? kMaxChunks : (uniform > L3 ? L3 : uniform);
        for (int c = 0; c <= n; c++) bound[c] = (int)((long)c * L3 / n);
        *plan_id = n;
        return n;
    }
    int cap = env_int_dropin("PLQCD_DROPIN_CAP", L3 / 8);
    cap = cap < 1 ? 1 : cap;
    int left[kMaxChunks], right[kMaxChunks], nl = 0, nr = 0, rem = L3, step = 1, k = 0;
    while (rem > 0 && nl + nr < kMaxChunks - 1) {
        int sz = step < cap ? step : cap;
        left[nl++] = sz < rem ? sz : rem;
        rem -= left[nl - 1];
        if (rem > 0) {
            right[nr++] = sz < rem ? sz : rem;
            rem -= right[nr - 1];
        }
        if (k++ > 0) step *= 2;  // 1, 1, 2, 4, ...
    }
    if (rem > 0) left[nl++] = rem;  // chunk budget exhausted: one more
    int n = 0;
    bound[0] = 0;
    for (int i = 0; i < nl; i++, n++) bound[n + 1] = bound[n] + left[i];
    for (int i = nr - 1; i >= 0; i--, n++) bound[n + 1] = bound[n] + right[i];
    *plan_id = -cap;
    return n;
}

uint64_t fingerprint(const su3 *u, long nlinks) {
    const uint64_t *w = reinterpret_cast<const uint64_t *>(u);
    long nwords = nlinks * 18;
    uint64_t h = 1469598103934665603ULL;
    const int samples = 1024;
    for (int k = 0; k < samples; k++) {
        long idx = (long)((double)k / samples * nwords);
        h = (h ^ w[idx]) * 1099511628211ULL;
    }
    h = (h ^ w[nwords - 1]) * 1099511628211ULL;
    return h;
}

// Whether the device copy `c` of link array `u` can serve this call:
//   PLQCD_GAUGE_CACHE unset: only a registered array, not marked dirty;
//   PLQCD_GAUGE_CACHE=1:     any array whose address and fingerprint match;
//   PLQCD_GAUGE_CACHE=0:     never.
// `fp` computes the fingerprint (only the sampled mode needs it).
template <class F>
bool keep_cached_gauge(const void *u, const LinkCache &c, uint64_t *new_fp, F fp) {
    const char *e = getenv("PLQCD_GAUGE_CACHE");
    if (e && *e == '0') return false;
    if (e && *e && *e != '0') {
        *new_fp = fp();
        return !c.dirty && c.u == u && c.fp == *new_fp;
    }
    return !c.dirty && c.u == u && g_registered == u;
}

// A call queues the upload of its links and waits once, at its end. A call
// that fails on the way waits as well (the caller gets its arrays back) and
// marks the device copy of the links it uses as not loaded.
struct CallGuard {
    LinkCache &links;
    bool ok = false;
    ~CallGuard() {
        if (ok) return;
        for (cudaStream_t st : {g_d.s_h2d, g_d.s_d2h, g_d.stream})
            if (st) cudaStreamSynchronize(st);
        cudaGetLastError();
        links.dirty = true;
    }
};

int ensure_locked() {
    if (!plqcd_g.init) return set_error(PLQCD_ERR_STATE, "hopping matrix called before init_plqcd");
    const int *L = plqcd_g.latdims;
    if (g_d.lat && memcmp(g_d.dims, L, sizeof g_d.dims) == 0) return PLQCD_OK;
    release_locked();
    int dev = 0;
    if (const char *e = getenv("PLQCD_DEVICE")) dev = atoi(e);
    cudaStream_t stream = nullptr;
    if (cudaSetDevice(dev) != cudaSuccess || cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        return set_error(PLQCD_ERR_CUDA, "drop-in: cannot create a stream on device %d", dev);
    }
    if (plqcd_lattice_create(L, dev, stream, &g_d.lat) != PLQCD_OK) {
        cudaStreamDestroy(stream);
        return plqcd_last_status();
    }
    g_d.stream = stream;
    memcpy(g_d.dims, L, sizeof g_d.dims);
    int rc = plqcd_gauge_create(g_d.lat, PLQCD_F64, 18, &g_d.gauge);
    if (rc != PLQCD_OK) {
        release_locked();
        return rc;
    }
    size_t bytes = spinor_parity_bytes(g_d.lat->geom.Vh, PLQCD_F64);
    void **bufs[4] = {&g_d.aos_in, &g_d.aos_out, &g_d.f_in, &g_d.f_out};
    for (void **b : bufs)
        if (cudaMalloc(b, bytes) != cudaSuccess) {
            cudaGetLastError();
            release_locked();
            return set_error(PLQCD_ERR_NOMEM, "drop-in: device allocation of %zu bytes failed", bytes);
        }
    bool ok = cudaStreamCreateWithFlags(&g_d.s_h2d, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&g_d.s_d2h, cudaStreamNonBlocking) == cudaSuccess;
    for (int c = 0; c < kMaxChunks && ok; c++)
        ok = cudaEventCreateWithFlags(&g_d.ev_in[c], cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreateWithFlags(&g_d.ev_out[c], cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreate(&g_d.ev_k0[c]) == cudaSuccess && cudaEventCreate(&g_d.ev_k1[c]) == cudaSuccess;
    for (cudaEvent_t *ev : {&g_d.ev_fork, &g_d.ev_join[0], &g_d.ev_join[1]})
        ok = ok && cudaEventCreateWithFlags(ev, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        release_locked();
        return set_error(PLQCD_ERR_CUDA, "drop-in: stream/event creation failed");
    }
    return PLQCD_OK;
}

// Enqueue the copy / compute pipeline of one call over chunks of t-slabs
// (contiguous half-site ranges). The host->device stream carries copies
// only, back to back, in the order last, 0, 1, ...; the compute stream
// converts each chunk to the device layout as it lands and computes the
// output chunk whose neighbours have all arrived; the device->host stream
// copies each output chunk back while later chunks are still in flight, so
// the two transfer directions overlap each other and the kernels.
// `capture`: kernel-time events become graph event-record nodes.
int enqueue_pipeline(plqcd_lattice *lat, const spinor *src, spinor *dst, int out_parity, unsigned flags, int nch,
                     const int *bound, bool capture) {
    const Geom &geo = lat->geom;
    cudaStream_t s = lat->stream;
    const int L3 = geo.L[3];
    const long slab = geo.Vh / L3;
    auto first = [&](int c) { return slab * (long)bound[c]; };
    auto count = [&](int c) { return first(c + 1) - first(c); };
    auto mark = [&](cudaEvent_t ev) {
        return capture ? cudaEventRecordWithFlags(ev, s, cudaEventRecordExternal) : cudaEventRecord(ev, s);
    };
    spinor *ain = static_cast<spinor *>(g_d.aos_in), *aout = static_cast<spinor *>(g_d.aos_out);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < nch && e == cudaSuccess; k++) {
        const int c = (k == 0) ? nch - 1 : k - 1;
        e = cudaMemcpyAsync(ain + first(c), src + first(c), count(c) * sizeof(spinor), cudaMemcpyHostToDevice,
                            g_d.s_h2d);
        if (e == cudaSuccess) e = cudaEventRecord(g_d.ev_in[c], g_d.s_h2d);
    }
    auto import = [&](int c) -> int {
        if (cudaStreamWaitEvent(s, g_d.ev_in[c], 0) != cudaSuccess)
            return set_error(PLQCD_ERR_CUDA, "hopping matrix: stream wait failed");
        // staging holds one parity, so it is addressed as parity 0
        return launch_spinor_import(geo, s, ain, 0, g_d.f_in, PLQCD_F64, first(c), count(c));
    };
    // Output chunk c is shifted one slab back from input chunk c: it covers
    // slabs [bound[c] - 1, bound[c+1] - 1) (chunk 0 starts at slab 0, the
    // last one ends at L3), whose neighbours lie in input chunks <= c and the
    // first-sent last chunk. It is computed as soon as input chunk c is in,
    // so results go back while the next input chunk is still coming up.
    auto out_first = [&](int c) { return c == 0 ? 0L : first(c) - slab; };
    auto out_end = [&](int c) { return c == nch - 1 ? geo.Vh : first(c + 1) - slab; };
    auto compute = [&](int c) -> int {
        const long h0 = out_first(c), n = out_end(c) - h0;
        mark(g_d.ev_k0[c]);
        if (n > 0) {
            DslashCall dc;
            dc.gauge = g_d.gauge->data;
            dc.prec = PLQCD_F64;
            dc.recon = 18;
            dc.out = g_d.f_out;
            dc.in = g_d.f_in;
            dc.out_parity = out_parity;
            dc.flags = flags;
            dc.h_begin = h0;
            dc.h_count = n;
            PLQCD_TRY(launch_dslash(geo, s, dc));
        }
        mark(g_d.ev_k1[c]);
        if (n <= 0) return PLQCD_OK;
        PLQCD_TRY(launch_spinor_export(geo, s, g_d.f_out, PLQCD_F64, 0, aout, h0, n));
        cudaError_t r = cudaEventRecord(g_d.ev_out[c], s);
        if (r == cudaSuccess) r = cudaStreamWaitEvent(g_d.s_d2h, g_d.ev_out[c], 0);
        if (r == cudaSuccess)
            r = cudaMemcpyAsync(dst + h0, aout + h0, n * sizeof(spinor), cudaMemcpyDeviceToHost, g_d.s_d2h);
        if (r != cudaSuccess) return set_error(PLQCD_ERR_CUDA, "hopping matrix: %s", cudaGetErrorString(r));
        return PLQCD_OK;
    };
    if (e == cudaSuccess) {
        if (nch > 1) PLQCD_TRY(import(nch - 1));
        for (int c = 0; c <= nch - 2; c++) {
            PLQCD_TRY(import(c));
            PLQCD_TRY(compute(c));
        }
        if (nch == 1) PLQCD_TRY(import(0));
        PLQCD_TRY(compute(nch - 1));
    }
    if (e != cudaSuccess) return set_error(PLQCD_ERR_CUDA, "hopping matrix: %s", cudaGetErrorString(e));
    return PLQCD_OK;
}

bool host_pinned(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

cudaGraphExec_t find_graph(const GraphKey &k) {
    for (int i = 0; i < kGraphSlots; i++)
        if (g_d.graph_exec[i] && g_d.graph_key[i] == k) return g_d.graph_exec[i];
    return nullptr;
}

// Capture the pipeline of `k` into a graph (fork to the copy streams and
// join back on the compute stream); nullptr when anything fails, and the
// caller runs the pipeline eagerly.
cudaGraphExec_t capture_graph(plqcd_lattice *lat, const GraphKey &k, const spinor *src, spinor *dst, int nch,
                              const int *bound) {
    cudaStream_t s = lat->stream;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    bool ok = cudaEventRecord(g_d.ev_fork, s) == cudaSuccess &&
              cudaStreamWaitEvent(g_d.s_h2d, g_d.ev_fork, 0) == cudaSuccess &&
              cudaStreamWaitEvent(g_d.s_d2h, g_d.ev_fork, 0) == cudaSuccess;
    ok = ok && enqueue_pipeline(lat, src, dst, k.parity, k.flags, nch, bound, true) == PLQCD_OK;
    ok = ok && cudaEventRecord(g_d.ev_join[0], g_d.s_h2d) == cudaSuccess &&
         cudaEventRecord(g_d.ev_join[1], g_d.s_d2h) == cudaSuccess &&
         cudaStreamWaitEvent(s, g_d.ev_join[0], 0) == cudaSuccess &&
         cudaStreamWaitEvent(s, g_d.ev_join[1], 0) == cudaSuccess;
    cudaGraph_t graph = nullptr;
    const bool ended = cudaStreamEndCapture(s, &graph) == cudaSuccess;
    cudaGraphExec_t exec = nullptr;
    if (ok && ended && graph && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) exec = nullptr;
    if (graph) cudaGraphDestroy(graph);
    if (!exec) {
        cudaGetLastError();
        clear_error();
        return nullptr;
    }
    const int slot = g_d.graph_next;
    g_d.graph_next = (slot + 1) % kGraphSlots;
    if (g_d.graph_exec[slot]) cudaGraphExecDestroy(g_d.graph_exec[slot]);
    g_d.graph_exec[slot] = exec;
    g_d.graph_key[slot] = k;
    return exec;
}

// out_parity 0: eo (qout even half from qin odd half); 1: oe.
double hop_call(spinor *qin, spinor *qout, su3 *u, int out_parity) {
    double t0 = stop_watch(0.0);
    clear_error();
    if (!qin || !qout || !u) {
        set_error(PLQCD_ERR_ARG, "hopping matrix: null argument");
        return -1.0;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (ensure_locked() != PLQCD_OK) return -1.0;
    plqcd_lattice *lat = g_d.lat;
    const long Vh = lat->geom.Vh;
    cudaStream_t s = lat->stream;
    if (cudaSetDevice(lat->device) != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "hopping matrix: cudaSetDevice failed");
        return -1.0;
    }
    g_d.h2d = g_d.d2h = 0;
    LinkCache &lc = g_d.links;
    CallGuard guard{lc};

    // gauge field: upload unless the device copy may serve (keep_cached_gauge)
    uint64_t fp = 0;
    if (!keep_cached_gauge(u, lc, &fp, [&] { return fingerprint(u, 8 * Vh); })) {
        if (upload_links(g_d.gauge, u) != PLQCD_OK) return -1.0;
        lc.u = u;
        lc.fp = fp;
        lc.dirty = false;
        g_d.h2d += 8.0 * Vh * sizeof(su3);
    }

    const int in_parity = out_parity ^ 1;
    const unsigned flags = env_flag("PLQCD_REF_COMPAT", false) ? PLQCD_DSLASH_COMPAT : 0u;
    int bound[kMaxChunks + 1], plan_id = 0;
    const int nch = chunk_plan(lat->geom.L[3], bound, &plan_id);
    const spinor *src = qin + in_parity * Vh;
    spinor *dst = qout + out_parity * Vh;

    // Replay the pipeline as one CUDA graph when the same host arrays come
    // back (the usual solver loop): one launch instead of ~10 API calls per
    // chunk. Captured on the second call with a key, so the first call has
    // tuned the kernels eagerly; pinned host arrays only.
    const GraphKey key{src, dst, out_parity, plan_id, flags, g_d.gauge->data};
    cudaGraphExec_t exec = nullptr;
    bool graphed = false;
    if (env_flag("PLQCD_DROPIN_GRAPH", true) && host_pinned(src) && host_pinned(dst)) {
        exec = find_graph(key);
        if (!exec && g_d.last_valid && g_d.last_key == key) exec = capture_graph(lat, key, src, dst, nch, bound);
        g_d.last_key = key;
        g_d.last_valid = true;
    }
    if (exec) {
        graphed = cudaGraphLaunch(exec, s) == cudaSuccess;
        if (!graphed) cudaGetLastError();
    }
    if (!graphed && enqueue_pipeline(lat, src, dst, out_parity, flags, nch, bound, false) != PLQCD_OK) return -1.0;
    cudaError_t e = cudaStreamSynchronize(g_d.s_d2h);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "hopping matrix: %s", cudaGetErrorString(e));
        return -1.0;
    }
    g_d.h2d += (double)Vh * sizeof(spinor);
    g_d.d2h += (double)Vh * sizeof(spinor);
    double kms = 0;
    for (int c = 0; c < nch; c++) {
        float ms = 0;
        cudaEventElapsedTime(&ms, g_d.ev_k0[c], g_d.ev_k1[c]);
        kms += ms;
    }
    g_d.kernel_ms = kms;
    lat->last_kernel_ms = kms;
    guard.ok = true;
    return stop_watch(t0);
}

// ---- split real / imaginary planes --------------------------------------------
// The reference's split-layout kernels (lib/dirac.c:2506, 4586, 7884, 9153)
// pack 2/4/8 x-sites per SIMD lane with their own site tables and gamma
// convention. This boundary keeps their names and argument order
// (qout_re, qout_im, u_re, u_im, qin_re, qin_im) but defines the split
// layout independently of any SIMD width: the API arrays with real and
// imaginary parts in separate planes, in even/odd site order,
//   qin_re[12*i + 3*spin + colour], u_re[9*(4*i + mu) + 3*row + col],
// and computes the same operator as the AoS entry points. With `short12`
// only link rows 0 and 1 are read and row 2 is rebuilt as
// conj(row0 x row1) (the reference's 2x3 variant, include/su3_intrin_
// highlevel_512.h:85-111, omits the conjugation).

uint64_t fingerprint_split(const double *re, const double *im, long n) {
    uint64_t h = 1469598103934665603ULL;
    const uint64_t *a = reinterpret_cast<const uint64_t *>(re), *b = reinterpret_cast<const uint64_t *>(im);
    for (int k = 0; k < 512; k++) {
        long idx = (long)((double)k / 512 * n);
        h = (h ^ a[idx]) * 1099511628211ULL;
        h = (h ^ b[idx]) * 1099511628211ULL;
    }
    return (h ^ a[n - 1] ^ (b[n - 1] << 1)) * 1099511628211ULL;
}

int load_gauge_split(plqcd_gauge *g, const double *ure, const double *uim) {
    const Geom &geo = g->lat->geom;
    cudaStream_t s = g->lat->stream;
    const long nlinks = 8 * geo.Vh, chunk = (long)(kStagingBytes / (18 * sizeof(double)));
    const long per = nlinks < chunk ? nlinks : chunk;
    std::lock_guard<std::mutex> lk(g->lat->staging_mu);
    void *stage = nullptr;
    PLQCD_TRY(lattice_staging(g->lat, sizeof(double) * 18 * per, &stage));
    double *st = static_cast<double *>(stage);
    for (long first = 0; first < nlinks; first += per) {
        const long n = nlinks - first < per ? nlinks - first : per;
        PLQCD_CUDA_TRY(cudaMemcpyAsync(st, ure + 9 * first, sizeof(double) * 9 * n, cudaMemcpyHostToDevice, s));
        PLQCD_CUDA_TRY(cudaMemcpyAsync(st + 9 * per, uim + 9 * first, sizeof(double) * 9 * n, cudaMemcpyHostToDevice, s));
        PLQCD_TRY(launch_gauge_import_split(geo, s, st, st + 9 * per, first, n, g->data, g->prec, g->recon));
    }
    return PLQCD_OK;
}

double hop_call_split(double *qout_re, double *qout_im, double *u_re, double *u_im, double *qin_re,
                      double *qin_im, int out_parity, bool short12) {
    double t0 = stop_watch(0.0);
    clear_error();
    if (!qout_re || !qout_im || !u_re || !u_im || !qin_re || !qin_im) {
        set_error(PLQCD_ERR_ARG, "split hopping matrix: null argument");
        return -1.0;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (ensure_locked() != PLQCD_OK) return -1.0;
    plqcd_lattice *lat = g_d.lat;
    const Geom &geo = lat->geom;
    const long Vh = geo.Vh;
    cudaStream_t s = lat->stream;
    if (cudaSetDevice(lat->device) != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "split hopping matrix: cudaSetDevice failed");
        return -1.0;
    }
    g_d.h2d = g_d.d2h = 0;
    LinkCache &lc = short12 ? g_d.split12 : g_d.split18;
    CallGuard guard{lc};
    plqcd_gauge *&gf = short12 ? g_d.gauge12 : g_d.gauge_split;
    if (!gf && plqcd_gauge_create(lat, PLQCD_F64, short12 ? 12 : 18, &gf) != PLQCD_OK) return -1.0;
    uint64_t fp = 0;
    // the split family registers its real-part plane u_re
    if (lc.im != u_im ||
        !keep_cached_gauge(u_re, lc, &fp, [&] { return fingerprint_split(u_re, u_im, 8 * Vh * 9); })) {
        if (load_gauge_split(gf, u_re, u_im) != PLQCD_OK) return -1.0;
        lc.u = u_re;
        lc.im = u_im;
        lc.fp = fp;
        lc.dirty = false;
        g_d.h2d += 2.0 * sizeof(double) * 9 * 8 * Vh;
    }
    const int in_parity = out_parity ^ 1;
    const size_t half = sizeof(double) * 12 * Vh;
    double *dre = static_cast<double *>(g_d.aos_in), *dim = dre + 12 * Vh;
    double *ore = static_cast<double *>(g_d.aos_out), *oim = ore + 12 * Vh;
    cudaError_t e = cudaMemcpyAsync(dre, qin_re + 12 * in_parity * Vh, half, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dim, qin_im + 12 * in_parity * Vh, half, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "split hopping matrix: H2D: %s", cudaGetErrorString(e));
        return -1.0;
    }
    if (launch_spinor_import_split(geo, s, dre, dim, g_d.f_in, PLQCD_F64) != PLQCD_OK) return -1.0;
    DslashCall dc;
    dc.gauge = gf->data;
    dc.prec = PLQCD_F64;
    dc.recon = gf->recon;
    dc.out = g_d.f_out;
    dc.in = g_d.f_in;
    dc.out_parity = out_parity;
    dc.flags = (env_flag("PLQCD_REF_COMPAT", false) && !short12) ? PLQCD_DSLASH_COMPAT : 0u;
    cudaEventRecord(g_d.ev_k0[0], s);
    if (launch_dslash(geo, s, dc) != PLQCD_OK) return -1.0;
    cudaEventRecord(g_d.ev_k1[0], s);
    if (launch_spinor_export_split(geo, s, g_d.f_out, PLQCD_F64, ore, oim) != PLQCD_OK) return -1.0;
    e = cudaMemcpyAsync(qout_re + 12 * out_parity * Vh, ore, half, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(qout_im + 12 * out_parity * Vh, oim, half, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "split hopping matrix: %s", cudaGetErrorString(e));
        return -1.0;
    }
    g_d.h2d += 2.0 * half;
    g_d.d2h += 2.0 * half;
    float ms = 0;
    cudaEventElapsedTime(&ms, g_d.ev_k0[0], g_d.ev_k1[0]);
    g_d.kernel_ms = ms;
    lat->last_kernel_ms = ms;
    guard.ok = true;
    return stop_watch(t0);
}

// ---- lane-packed types (include/su3_256.h, su3_512.h) ----------------------------
// The reference's intrin_256 / intrin_512 / single_mic kernels
// (lib/dirac.c:3506, 7122, 7503) take arrays of packed objects that each
// hold `lanes` (2 or 4) consecutive even/odd sites, one complex element of
// every site per lane (tests/test_hopping.c:256-275): complex element e of
// site s sits at ((s / lanes) * E + e) * lanes + s % lanes, E = 12 for a
// spinor and 36 for the four links of a site. The arrays are moved as they
// are and unpacked / packed on the device around the same kernels as the
// AoS entry points; the result is the correct operator for every name.

__global__ void k_lanes_to_sites(double2 *dst, const double2 *src, long nsites, int lanes, int E) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= nsites * E) return;
    const long site = i / E;
    const int e = (int)(i - site * E);
    dst[i] = src[((site / lanes) * E + e) * lanes + site % lanes];
}

__global__ void k_sites_to_lanes(double2 *dst, const double2 *src, long nsites, int lanes, int E) {
    const long j = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (j >= nsites * E) return;
    const int lane = (int)(j % lanes);
    const long rest = j / lanes;
    const int e = (int)(rest % E);
    const long site = (rest / E) * lanes + lane;
    dst[j] = src[site * E + e];
}

int relayout(cudaStream_t s, void *dst, const void *src, long nsites, int lanes, int E, bool to_sites) {
    const long n = nsites * E;
    if (n == 0) return PLQCD_OK;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (to_sites)
        k_lanes_to_sites<<<blocks, 256, 0, s>>>(static_cast<double2 *>(dst), static_cast<const double2 *>(src),
                                                 nsites, lanes, E);
    else
        k_sites_to_lanes<<<blocks, 256, 0, s>>>(static_cast<double2 *>(dst), static_cast<const double2 *>(src),
                                                 nsites, lanes, E);
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

// gauge field from a lane-packed host array, in chunks of whole packed objects
int load_gauge_packed(plqcd_gauge *g, const void *u, int lanes) {
    const Geom &geo = g->lat->geom;
    cudaStream_t s = g->lat->stream;
    const long nsites = 2 * geo.Vh, chunk = (long)(kStagingBytes / (2 * 4 * sizeof(su3))) & ~3L;
    const long per = nsites < chunk ? nsites : chunk;
    std::lock_guard<std::mutex> lk(g->lat->staging_mu);
    void *st = nullptr;
    PLQCD_TRY(lattice_staging(g->lat, 2 * per * 4 * sizeof(su3), &st));
    char *packed = static_cast<char *>(st), *aos = packed + per * 4 * sizeof(su3);
    for (long first = 0; first < nsites; first += per) {
        const long n = nsites - first < per ? nsites - first : per;
        PLQCD_CUDA_TRY(cudaMemcpyAsync(packed, static_cast<const char *>(u) + first * 4 * sizeof(su3),
                                       n * 4 * sizeof(su3), cudaMemcpyHostToDevice, s));
        PLQCD_TRY(relayout(s, aos, packed, n, lanes, 36, true));
        PLQCD_TRY(launch_gauge_import(geo, s, aos, 4 * first, 4 * n, g->data, g->prec, g->recon));
    }
    return PLQCD_OK;
}

double hop_call_packed(const void *qin, void *qout, const void *u, int out_parity, int lanes, bool short12) {
    double t0 = stop_watch(0.0);
    clear_error();
    if (!qin || !qout || !u) {
        set_error(PLQCD_ERR_ARG, "packed hopping matrix: null argument");
        return -1.0;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    if (ensure_locked() != PLQCD_OK) return -1.0;
    plqcd_lattice *lat = g_d.lat;
    const Geom &geo = lat->geom;
    const long Vh = geo.Vh;
    cudaStream_t s = lat->stream;
    if (Vh % lanes) {
        set_error(PLQCD_ERR_ARG, "packed hopping matrix: half volume %ld is not a multiple of %d lanes", Vh, lanes);
        return -1.0;
    }
    if (cudaSetDevice(lat->device) != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "packed hopping matrix: cudaSetDevice failed");
        return -1.0;
    }
    g_d.h2d = g_d.d2h = 0;
    LinkCache &lc = short12 ? g_d.packed12 : g_d.packed18;
    CallGuard guard{lc};
    plqcd_gauge *&gf = short12 ? g_d.gauge_packed12 : g_d.gauge_packed;
    if (!gf && plqcd_gauge_create(lat, PLQCD_F64, short12 ? 12 : 18, &gf) != PLQCD_OK) return -1.0;
    uint64_t fp = 0;
    if (lc.lanes != lanes ||
        !keep_cached_gauge(u, lc, &fp, [&] { return fingerprint(static_cast<const su3 *>(u), 8 * Vh); })) {
        if (load_gauge_packed(gf, u, lanes) != PLQCD_OK) return -1.0;
        lc.u = u;
        lc.lanes = lanes;
        lc.fp = fp;
        lc.dirty = false;
        g_d.h2d += 8.0 * Vh * sizeof(su3);
    }
    const int in_parity = out_parity ^ 1;
    const size_t half = sizeof(spinor) * Vh;  // one parity, in either layout
    void *stage = g_d.aos_out, *aos = g_d.aos_in;
    cudaError_t e = cudaMemcpyAsync(stage, static_cast<const char *>(qin) + in_parity * half, half,
                                    cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "packed hopping matrix: H2D: %s", cudaGetErrorString(e));
        return -1.0;
    }
    if (relayout(s, aos, stage, Vh, lanes, 12, true) != PLQCD_OK) return -1.0;
    if (launch_spinor_import(geo, s, aos, 0, g_d.f_in, PLQCD_F64, 0, Vh) != PLQCD_OK) return -1.0;
    DslashCall dc;
    dc.gauge = gf->data;
    dc.prec = PLQCD_F64;
    dc.recon = gf->recon;
    dc.out = g_d.f_out;
    dc.in = g_d.f_in;
    dc.out_parity = out_parity;
    cudaEventRecord(g_d.ev_k0[0], s);
    if (launch_dslash(geo, s, dc) != PLQCD_OK) return -1.0;
    cudaEventRecord(g_d.ev_k1[0], s);
    if (launch_spinor_export(geo, s, g_d.f_out, PLQCD_F64, 0, aos, 0, Vh) != PLQCD_OK) return -1.0;
    if (relayout(s, stage, aos, Vh, lanes, 12, false) != PLQCD_OK) return -1.0;
    e = cudaMemcpyAsync(static_cast<char *>(qout) + out_parity * half, stage, half, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error(PLQCD_ERR_CUDA, "packed hopping matrix: %s", cudaGetErrorString(e));
        return -1.0;
    }
    g_d.h2d += (double)half;
    g_d.d2h += (double)half;
    float ms = 0;
    cudaEventElapsedTime(&ms, g_d.ev_k0[0], g_d.ev_k1[0]);
    g_d.kernel_ms = ms;
    lat->last_kernel_ms = ms;
    guard.ok = true;
    return stop_watch(t0);
}

}  // namespace

namespace plqcd {
// finalize_plqcd: drop every device copy and the registration (a later
// array at the same host address is a different field)
void dropin_release() {
    std::lock_guard<std::mutex> lk(g_mu);
    release_locked();
    g_registered = nullptr;
}
}  // namespace plqcd

extern "C" int plqcd_gauge_update(const su3 *u) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_registered = u;
    for (LinkCache *c : {&g_d.links, &g_d.split18, &g_d.split12, &g_d.packed18, &g_d.packed12}) c->dirty = true;
    return PLQCD_OK;
}

// split-layout names: include/dirac.h:31-32 (SSE3), 39-40 (AVX), 55-62 (MIC)
#define PLQCD_SPLIT_ENTRY(name, parity, short12)                                                               \
    extern "C" double name(double *qout_re, double *qout_im, double *u_re, double *u_im, double *qin_re,       \
                           double *qin_im) {                                                                   \
        return hop_call_split(qout_re, qout_im, u_re, u_im, qin_re, qin_im, parity, short12);                  \
    }
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_eo_sse3_intrin_nohalfspinor, 0, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_oe_sse3_intrin_nohalfspinor, 1, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_eo_avx_nohalfspinor, 0, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_oe_avx_nohalfspinor, 1, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_eo_single_mic_split, 0, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_oe_single_mic_split, 1, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_eo_single_mic_split_nohalfspinor, 0, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_oe_single_mic_split_nohalfspinor, 1, false)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_eo_single_mic_split_nohalfspinor_short, 0, true)
PLQCD_SPLIT_ENTRY(plqcd_hopping_matrix_oe_single_mic_split_nohalfspinor_short, 1, true)
#undef PLQCD_SPLIT_ENTRY

extern "C" int plqcd_dropin_last_stats(double *kernel_ms, double *h2d, double *d2h) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (kernel_ms) *kernel_ms = g_d.kernel_ms;
    if (h2d) *h2d = g_d.h2d;
    if (d2h) *d2h = g_d.d2h;
    return PLQCD_OK;
}

// lib/dirac.c:35 and :414, plus the same-signature SSE3 names of
// lib/dirac.c:801, 1272, 1748, 2124.
extern "C" double plqcd_hopping_matrix_eo_sse3_assymbly(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 0);
}
extern "C" double plqcd_hopping_matrix_oe_sse3_assymbly(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 1);
}
extern "C" double plqcd_hopping_matrix_eo_sse3_intrin(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 0);
}
extern "C" double plqcd_hopping_matrix_oe_sse3_intrin(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 1);
}
extern "C" double plqcd_hopping_matrix_eo_sse3_intrin_blocking(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 0);
}
extern "C" double plqcd_hopping_matrix_oe_sse3_intrin_blocking(spinor *qin, spinor *qout, su3 *u) {
    return hop_call(qin, qout, u, 1);
}

// lane-packed names: include/dirac.h:37-38 (256), 46-51 (512, MIC); the
// _short form reads link rows 0 and 1 and rebuilds row 2 as conj(row0 x row1)
extern "C" double plqcd_hopping_matrix_eo_intrin_256(spinor_256 *qin, spinor_256 *qout, su3_256 *u) {
    return hop_call_packed(qin, qout, u, 0, 2, false);
}
extern "C" double plqcd_hopping_matrix_oe_intrin_256(spinor_256 *qin, spinor_256 *qout, su3_256 *u) {
    return hop_call_packed(qin, qout, u, 1, 2, false);
}
extern "C" double plqcd_hopping_matrix_eo_intrin_512(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 0, 4, false);
}
extern "C" double plqcd_hopping_matrix_oe_intrin_512(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 1, 4, false);
}
extern "C" double plqcd_hopping_matrix_eo_single_mic(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 0, 4, false);
}
extern "C" double plqcd_hopping_matrix_oe_single_mic(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 1, 4, false);
}
extern "C" double plqcd_hopping_matrix_eo_single_mic_short(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 0, 4, true);
}
extern "C" double plqcd_hopping_matrix_oe_single_mic_short(spinor_512 *qin, spinor_512 *qout, su3_512 *u) {
    return hop_call_packed(qin, qout, u, 1, 4, true);
}
