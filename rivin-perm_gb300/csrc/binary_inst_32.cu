// Instantiations of binary_glynn_kernel with 32 padded rows: row groups G in
// {5, 6, 7, 8, 10}.
#include "binary_glynn.cuh"

namespace pg {

cudaError_t launch_binary_npad32(int G, const BinaryArgs &args, int blocks, cudaStream_t stream) {
    switch (G) {
        case 5: return launch_binary_glynn<32, 5>(args, blocks, stream);
        case 6: return launch_binary_glynn<32, 6>(args, blocks, stream);
        case 7: return launch_binary_glynn<32, 7>(args, blocks, stream);
        case 8: return launch_binary_glynn<32, 8>(args, blocks, stream);
        case 10: return launch_binary_glynn<32, 10>(args, blocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
