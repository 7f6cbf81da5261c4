// Sweep kernels for the D2Q9 descriptor, FP16-shifted storage: every launch shape,
// parity and collision variant, and the multi-step tiles.
#include "sweep_launch.cuh"

namespace kel {
namespace gb {
template cudaError_t launch_sweep_part<D2Q9, PART_FP16S>(const SweepParams &, bool, int, cudaStream_t);
template cudaError_t launch_tile_part<PART_FP16S>(const TileParams &, int, bool, cudaStream_t);
} // namespace gb
} // namespace kel
