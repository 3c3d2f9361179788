// Quantise + pack of fp16, with the half arithmetic of the reference's half kernels activations.
#include "pack_tile.cuh"

namespace exb {
template int launch_pack_bits<HalfBits>(const PackParams&, int, const TileShape&, cudaStream_t);
}
