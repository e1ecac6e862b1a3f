// Test-only: the absorbed backward with a way to set its status word, as if a wait of an earlier launch had run out.
#include "absorbed_backward.cu"

extern "C" int dscuda_test_set_absorbed_backward_status(int status) {
    return cudaMemcpyToSymbol(dscuda::absorbed_backward_status, &status, sizeof(int)) == cudaSuccess ? 0 : 1;
}

// t: dquery, dquery_rope, dlatent, dkey_rope, dout, output, lse, query, query_rope, latent, key_rope
extern "C" int dscuda_test_absorbed_backward(void** t, int batch, int sequence, int heads, float scale, void* stream) {
    using bf16 = __nv_bfloat16;
    auto tensor = [&](int i) { return static_cast<bf16*>(t[i]); };
    try {
        dscuda::mla_compressed_attention_backward_cuda(tensor(0), tensor(1), tensor(2), tensor(3), tensor(4), tensor(5), static_cast<const float*>(t[6]), tensor(7),
                                                       tensor(8), tensor(9), tensor(10), batch, sequence, heads, 512, 64, scale, static_cast<cudaStream_t>(stream));
    } catch (const std::exception&) {
        return 1;
    }
    return 0;
}
