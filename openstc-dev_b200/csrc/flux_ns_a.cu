// flux_ns_a.cu — the flux kernel family (flux.cuh) for mechanisms of
// 1, 2, 3, 4, 5 species, in its 128-register budget only (the
// 9-species unit flux9.cu carries every budget the autotuner chooses from).
#include "common.cuh"

namespace ostc {
// this unit's copy of the run parameters (written by upload_param) and of
// the zone table of tile-table launches (written by upload_zones)
static __constant__ DevParam c_p;
}  // namespace ostc

#include "kernels.cuh"

namespace ostc {
static __constant__ DevZone c_zones[kMaxTableZones];
}  // namespace ostc

#define OSTC_FLUX_REDUCED
#include "flux.cuh"

namespace ostc {

template cudaError_t launch_flux_nt<1, 0>(const DevZone &, int, int, const TileShape &, const FluxTable *, int,
                                           int, int, cudaStream_t);
template cudaError_t launch_flux_nt<2, 0>(const DevZone &, int, int, const TileShape &, const FluxTable *, int,
                                           int, int, cudaStream_t);
template cudaError_t launch_flux_nt<3, 0>(const DevZone &, int, int, const TileShape &, const FluxTable *, int,
                                           int, int, cudaStream_t);
template cudaError_t launch_flux_nt<4, 0>(const DevZone &, int, int, const TileShape &, const FluxTable *, int,
                                           int, int, cudaStream_t);
template cudaError_t launch_flux_nt<5, 0>(const DevZone &, int, int, const TileShape &, const FluxTable *, int,
                                           int, int, cudaStream_t);

cudaError_t upload_param_flux_ns_a(const DevParam &p, cudaStream_t s) {
  return cudaMemcpyToSymbolAsync(c_p, &p, sizeof(DevParam), 0, cudaMemcpyHostToDevice, s);
}

cudaError_t upload_zones_flux_ns_a(const DevZone *z, int n, cudaStream_t s) {
  if (n < 0 || n > kMaxTableZones) return cudaErrorInvalidValue;
  return n ? cudaMemcpyToSymbolAsync(c_zones, z, sizeof(DevZone) * n, 0, cudaMemcpyHostToDevice, s) : cudaSuccess;
}

}  // namespace ostc
