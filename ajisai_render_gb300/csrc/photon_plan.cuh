// How the photons of an SPPM render are cut into waves (host code, used by
// sppm.cu).
#pragma once
#include <algorithm>
#include <cstdint>

namespace ajg {

// Deposit records a wave holds (48 + 4 bytes each), and the photons of waves
// of several iterations.
constexpr uint64_t kDepositRecords = 1ull << 25;
constexpr uint64_t kWavePhotons = 1ull << 21;

struct PhotonPlan {
  uint64_t chunk;    // photons of an iteration in a wave
  uint64_t group;    // iterations in a wave
  uint64_t depths;   // depths whose deposits are recorded before a join
  uint64_t records;  // deposits of an iteration before a join, at most
};

// An iteration's photons go in equal chunks of at most `wave_paths`.  A photon
// deposits once per depth from 2 on: where the record buffer holds an
// iteration's deposits of all depths, they are joined with the visible points
// once, and a wave takes several iterations, as many as fill the GPU and the
// buffer; where it does not, after every `depths` depths that it holds.
// (Chunks cut down to what fits with all depths, the form before: each ran all
// depths' launches and a join of its own, and 2 M photons of the sphere took
// 529 ms at a depth limit of 1,024 and 24 ms at 128.)
// `tries`: allocations that failed.  After one an iteration goes alone, then
// the chunks and the buffer are halved each time.
inline PhotonPlan photon_plan(uint64_t photons, uint64_t iterations,
                              int max_depth, uint64_t wave_paths, int tries) {
  PhotonPlan p{1, 1, 0, 0};
  const int halved = tries > 1 ? tries - 1 : 0;
  const uint64_t budget = kDepositRecords >> halved;
  const uint64_t most =
      std::max<uint64_t>(1, std::min(photons, wave_paths) >> halved);
  const uint64_t n_chunks = (photons + most - 1) / most;
  if (n_chunks) p.chunk = (photons + n_chunks - 1) / n_chunks;
  const uint64_t dep = max_depth > 1 ? (uint64_t)max_depth - 1 : 0;
  p.depths = std::min(dep, std::max<uint64_t>(1, budget / p.chunk));
  p.records = p.chunk * p.depths;
  if (n_chunks == 1 && tries == 0 && p.depths == dep) {
    uint64_t fit = std::min(wave_paths, kWavePhotons) / p.chunk;
    if (dep) fit = std::min(fit, budget / p.records);
    p.group = std::max<uint64_t>(1, std::min(fit, iterations));
    const uint64_t waves = (iterations + p.group - 1) / p.group;
    if (waves) p.group = (iterations + waves - 1) / waves;
  }
  return p;
}

}  // namespace ajg
