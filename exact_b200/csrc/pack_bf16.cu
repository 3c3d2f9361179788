// Quantise + pack of bf16 activations.
#include "pack_tile.cuh"

namespace exb {
template int launch_pack_bits<uint16_t>(const PackParams&, int, const TileShape&, cudaStream_t);
}
