// The step between the q | k | v projection and attention: rotary embedding of the new token's query and key
// (rotate-half on the first rotary_dim channels, mega_kernel_qwen36/reference.py:91-114) and the append of its
// key and value to the caches, in one launch.
//
// A few tens of KB: all latency.  One CTA per (token, head) and a thread per channel, so every load is issued
// at once; as separate tensor operations the same work was a dozen launches of about 2 us each.
#include "mk36_common.cuh"

namespace mk36 {

struct AppendParams {
    const void* qkv;   // [B][(Hq + 2 Hkv) * D]
    const float* cos;  // [rotary] or null: no rotation
    const float* sin;
    void* q;           // [B][Hq][D]
    void* k_cache;     // [B][capacity][Hkv][D]
    void* v_cache;
    int Hq, Hkv, D, rotary;
    size_t position, capacity;
};

template <typename T>
__global__ void __launch_bounds__(256) attention_append_kernel(const AppendParams p) {
    const int heads = p.Hq + 2 * p.Hkv;
    const int b = blockIdx.x / heads, h = blockIdx.x - b * heads;
    const T* src = static_cast<const T*>(p.qkv) + (size_t)blockIdx.x * p.D;
    T* dst;
    if (h < p.Hq) {
        dst = static_cast<T*>(p.q) + ((size_t)b * p.Hq + h) * p.D;
    } else {
        const bool is_k = h < p.Hq + p.Hkv;
        const int kh = h - p.Hq - (is_k ? 0 : p.Hkv);
        dst = static_cast<T*>(is_k ? p.k_cache : p.v_cache) + (((size_t)b * p.capacity + p.position) * p.Hkv + kh) * p.D;
    }
    const int half = p.rotary / 2;
    for (int d = threadIdx.x; d < p.D; d += blockDim.x) {
        T v = src[d];
        if (p.cos && d < p.rotary && h < p.Hq + p.Hkv) {
            // the partner is (-second half, first half); products and sum are rounded one by one, as tensor operations round
            const float turned = d < p.rotary - half ? -to_float<T>(src[half + d]) : to_float<T>(src[d - (p.rotary - half)]);
            v = from_float<T>(__fadd_rn(__fmul_rn(to_float<T>(v), p.cos[d]), __fmul_rn(turned, p.sin[d])));
        }
        dst[d] = v;
    }
}

}  // namespace mk36

using namespace mk36;

extern "C" int mk36_attention_append(const mk36_attention_append_args* a, void* stream) {
    if (!a) MK36_FAIL(MK36_ERR_INVALID_ARG, "attention_append: args is NULL");
    if (!a->qkv || !a->q || !a->k_cache || !a->v_cache || (a->cos && !a->sin)) MK36_FAIL(MK36_ERR_INVALID_ARG, "attention_append: NULL tensor pointer");
    if (a->batch <= 0 || a->query_heads <= 0 || a->kv_heads <= 0 || a->head_dim <= 0 || a->capacity <= 0)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "attention_append: sizes must be positive");
    if (a->position < 0 || a->position >= a->capacity) MK36_FAIL(MK36_ERR_INVALID_ARG, "attention_append: position must lie inside the cache");
    if (a->cos && (a->rotary_dim <= 0 || a->rotary_dim > a->head_dim)) MK36_FAIL(MK36_ERR_INVALID_ARG, "attention_append: rotary_dim must be in [1, head_dim]");
    const long long ctas = (long long)a->batch * (a->query_heads + 2ll * a->kv_heads);
    if (ctas > 0x7fffffffLL) MK36_FAIL(MK36_ERR_UNSUPPORTED, "attention_append: too many heads");
    AppendParams p;
    p.qkv = a->qkv;
    p.cos = a->cos;
    p.sin = a->sin;
    p.q = a->q;
    p.k_cache = a->k_cache;
    p.v_cache = a->v_cache;
    p.Hq = a->query_heads;
    p.Hkv = a->kv_heads;
    p.D = a->head_dim;
    p.rotary = a->cos ? a->rotary_dim : 0;
    p.position = (size_t)a->position;
    p.capacity = (size_t)a->capacity;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned threads = a->head_dim >= 256 ? 256u : (unsigned)(a->head_dim + 31) / 32 * 32;
    switch (a->dtype) {
        case MK36_BF16: attention_append_kernel<__nv_bfloat16><<<(unsigned)ctas, threads, 0, s>>>(p); break;
        case MK36_F16: attention_append_kernel<__half><<<(unsigned)ctas, threads, 0, s>>>(p); break;
        case MK36_F32: attention_append_kernel<float><<<(unsigned)ctas, threads, 0, s>>>(p); break;
        default: MK36_FAIL(MK36_ERR_UNSUPPORTED, "attention_append: unsupported dtype %d", a->dtype);
    }
    MK36_CUDA_OK(cudaGetLastError());
    return MK36_OK;
}
