// Instantiations of binary_glynn_kernel with 24 padded rows: row groups G in
// {5, 6, 7, 8, 10}.
#include "binary_glynn.cuh"

namespace pg {

cudaError_t launch_binary_npad24(int G, const BinaryArgs &args, int blocks, cudaStream_t stream) {
    switch (G) {
        case 5: return launch_binary_glynn<24, 5>(args, blocks, stream);
        case 6: return launch_binary_glynn<24, 6>(args, blocks, stream);
        case 7: return launch_binary_glynn<24, 7>(args, blocks, stream);
        case 8: return launch_binary_glynn<24, 8>(args, blocks, stream);
        case 10: return launch_binary_glynn<24, 10>(args, blocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_binary_npad28(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad32(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad36(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad40(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad44(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);
cudaError_t launch_binary_npad48(int G, const BinaryArgs &args, int blocks, cudaStream_t stream);

int binary_npad(int n) { return n < 24 || n > 48 ? 0 : (n + 3) & ~3; }

bool binary_compiled(int NPAD, int G) {
    const bool g = G == 5 || G == 6 || G == 7 || G == 8 || G == 10;
    return NPAD >= 24 && NPAD <= 48 && NPAD % 4 == 0 && g;
}

cudaError_t launch_binary_any(int NPAD, int G, const BinaryArgs &args, int blocks,
                              cudaStream_t stream) {
    switch (NPAD) {
        case 24: return launch_binary_npad24(G, args, blocks, stream);
        case 28: return launch_binary_npad28(G, args, blocks, stream);
        case 32: return launch_binary_npad32(G, args, blocks, stream);
        case 36: return launch_binary_npad36(G, args, blocks, stream);
        case 40: return launch_binary_npad40(G, args, blocks, stream);
        case 44: return launch_binary_npad44(G, args, blocks, stream);
        case 48: return launch_binary_npad48(G, args, blocks, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
