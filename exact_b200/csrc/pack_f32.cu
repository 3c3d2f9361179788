// Quantise + pack of fp32 activations.
#include "pack_tile.cuh"

namespace exb {
template int launch_pack_bits<float>(const PackParams&, int, const TileShape&, cudaStream_t);
}
