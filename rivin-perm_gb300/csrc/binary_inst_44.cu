// Instantiations of binary_glynn_kernel with 44 padded rows: row groups G in
// {5, 6, 7, 8, 10}.
#include "binary_glynn.cuh"

namespace pg {

cudaError_t launch_binary_npad44(int G, const BinaryArgs &args, int blocks, cudaStream_t stream) {
    switch (G) {
        case 5: return launch_binary_glynn<44, 5>(args, blocks, stream);
        case 6: return launch_binary_glynn<44, 6>(args, blocks, stream);
        case 7: return launch_binary_glynn<44, 7>(args, blocks, stream);
        case 8: return launch_binary_glynn<44, 8>(args, blocks, stream);
        case 10: return launch_binary_glynn<44, 10>(args, blocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
