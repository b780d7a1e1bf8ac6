// tune.h -- launch-configuration autotuner (tune.cpp).
#pragma once

#include <cuda_runtime.h>
#include <unistd.h>

#include <functional>
#include <string>
#include <vector>

namespace plqcd {

struct TuneResult {
    int variant = 0;  // kernel-family specific (e.g. load strategy)
    int block = 128;
    double ms = 0.0;
};

bool tune_enabled();
// run(config, trial): launch one configuration; trial launches must write
// only to scratch outputs (they are repeated while timing).
int tune_launch(const std::string &key, cudaStream_t s, const std::vector<TuneResult> &cands,
                const std::function<int(const TuneResult &, bool)> &run);
// "<device name>|" prefix for keys, so cache files do not mix GPU models
const std::string &device_tag();
// end of every key: the number of the families' candidate lists, raised when
// they gain kernels
constexpr char kTuneListTag[] = "|c2";
bool tune_lookup(const std::string &key, TuneResult *out);

// What tells the launches of the tuned families apart, as numbers: the look-up
// of a launch that is already tuned needs no key text and no candidate list
// (a hop of a 4x6x8x10 lattice runs 4 us on the device; building them took
// 2 us, 18 with the tile plans of the TMA candidates).
struct TuneId {
    int v[12];  // device, family, precision, reconstruction, mode bits, RHS, extents (the rest 0)
    bool operator==(const TuneId &o) const;
};
enum TuneFamily : int { kTuneDslash = 1, kTuneMrhs = 2 };
TuneId tune_id(TuneFamily family, int prec, int recon, int mode, int nrhs, const int dims[4]);
// the tuned configuration of `id`, once tune_remember has tied it to the
// entry of `key` (no effect while there is no such entry); dropped when
// entries are cleared or loaded
bool tune_recall(const TuneId &id, TuneResult *out);
void tune_remember(const TuneId &id, const std::string &key);

}  // namespace plqcd
