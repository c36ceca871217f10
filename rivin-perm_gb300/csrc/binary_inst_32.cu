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

cudaError_t launch_binary_npad40(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad48(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);

int binary_npad(int n) { return n <= 32 ? 32 : n <= 40 ? 40 : n <= 48 ? 48 : 0; }

bool binary_compiled(int NPAD, int G) {
    const bool g = G == 5 || G == 6 || G == 7 || G == 8 || G == 10;
    return (NPAD == 32 || NPAD == 40 || NPAD == 48) && g;
}

cudaError_t launch_binary_any(int NPAD, int G, const BinaryArgs &args, int blocks,
                              cudaStream_t stream) {
    if (!binary_compiled(NPAD, G)) return cudaErrorInvalidValue;
    return NPAD == 32 ? launch_binary_npad32(G, args, blocks, stream)
         : NPAD == 40 ? launch_binary_npad40(G, args, blocks, stream)
                      : launch_binary_npad48(G, args, blocks, stream);
}

}  // namespace pg
