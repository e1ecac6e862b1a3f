// Test-only: the projection kernels with a way to set their status word, as if a wait of an earlier launch had run out.
#include "projection_gemm.cu"

extern "C" int dscuda_test_set_projection_status(int status) {
    return cudaMemcpyToSymbol(dscuda::projection_status, &status, sizeof(int)) == cudaSuccess ? 0 : 1;
}

extern "C" int dscuda_test_up_project(void* k_nope, void* v, const void* latent, const void* w_uk, const void* w_uv, long long rows, int heads, void* stream) {
    using bf16 = __nv_bfloat16;
    try {
        dscuda::mla_up_project_cuda(static_cast<bf16*>(k_nope), static_cast<bf16*>(v), static_cast<const bf16*>(latent), static_cast<const bf16*>(w_uk),
                                    static_cast<const bf16*>(w_uv), rows, heads, static_cast<cudaStream_t>(stream));
    } catch (const std::exception&) {
        return 1;
    }
    return 0;
}
