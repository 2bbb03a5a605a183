// Linear-attention recurrent decode step for sm_100a.
//
//   S'[kd, vd] = decay * S[kd, vd] + k[kd] * (beta * v[vd])        (fp32 state)
//   out[vd]    = sum_kd q[kd] * S'[kd, vd]
//
// One CTA owns a slice of 32 value columns of one (batch, value head) state matrix, so at batch
// 1 with 32 heads x 128 columns there are 128 CTAs (the reference's kernel, a thread per output
// column with a serial loop over kd, runs 16: csrc/linear_attention_decode.cu:10-42, 77).  Aligned shapes
// run the strip kernels further down; linear_attention_kernel takes the others.
// The state update uses separately rounded multiply / add (no FMA contraction) so that the new
// state is bit-identical to reference.py:164 (`state.mul(decay) + einsum(k, v)`).
#include "mk36_common.cuh"

namespace mk36 {

constexpr int kLinThreads = 256;
constexpr int kLinCols = 32;

struct LinParams {
    const void* q;
    const void* k;
    const void* v;
    const float* state;
    void* out;
    float* new_state;
    const float* decay_ph;
    const float* beta_ph;
    int B, Hk, Hv, Dk, Dv;
    float decay;
};

template <typename T, int VEC>
__global__ void __launch_bounds__(kLinThreads) linear_attention_kernel(const LinParams p) {
    constexpr int CT = kLinCols / VEC;     // threads across the column slice
    constexpr int RG = kLinThreads / CT;   // row groups
    extern __shared__ float s_dyn[];       // q[Dk], k[Dk]
    __shared__ float s_red[RG][kLinCols + 1];

    const int slices = (p.Dv + kLinCols - 1) / kLinCols;
    const int slice = blockIdx.x % slices;
    const int bh = blockIdx.x / slices;
    const int h = bh % p.Hv;
    const int b = bh / p.Hv;
    const int hk = h / (p.Hv / p.Hk);

    float* s_q = s_dyn;
    float* s_k = s_dyn + p.Dk;
    const T* q = static_cast<const T*>(p.q) + ((size_t)b * p.Hk + hk) * p.Dk;
    const T* k = static_cast<const T*>(p.k) + ((size_t)b * p.Hk + hk) * p.Dk;
    for (int i = threadIdx.x; i < p.Dk; i += kLinThreads) {
        s_q[i] = to_float<T>(q[i]);
        s_k[i] = to_float<T>(k[i]);
    }

    const int ct = threadIdx.x % CT;
    const int rg = threadIdx.x / CT;
    const int col0 = slice * kLinCols + ct * VEC;
    const float decay = p.decay_ph ? p.decay_ph[(size_t)b * p.Hv + h] : p.decay;
    const float beta = p.beta_ph ? p.beta_ph[(size_t)b * p.Hv + h] : 1.0f;
    const T* v = static_cast<const T*>(p.v) + ((size_t)b * p.Hv + h) * p.Dv;

    float vv[VEC], o[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        const float raw = (col0 + j < p.Dv) ? to_float<T>(v[col0 + j]) : 0.0f;
        vv[j] = p.beta_ph ? __fmul_rn(raw, beta) : raw;
        o[j] = 0.0f;
    }
    __syncthreads();

    const size_t base = ((size_t)b * p.Hv + h) * p.Dk * p.Dv;
    const float* src = p.state + base;
    float* dst = p.new_state + base;

    if (VEC == 4) {
        if (col0 < p.Dv) {  // Dv % 4 == 0 on this path, so the whole float4 is in range
#pragma unroll 4
            for (int kd = rg; kd < p.Dk; kd += RG) {
                const float4 s = *reinterpret_cast<const float4*>(src + (size_t)kd * p.Dv + col0);
                const float kk = s_k[kd], qq = s_q[kd];
                float4 n;
                n.x = __fadd_rn(__fmul_rn(s.x, decay), __fmul_rn(kk, vv[0]));
                n.y = __fadd_rn(__fmul_rn(s.y, decay), __fmul_rn(kk, vv[1 % VEC]));
                n.z = __fadd_rn(__fmul_rn(s.z, decay), __fmul_rn(kk, vv[2 % VEC]));
                n.w = __fadd_rn(__fmul_rn(s.w, decay), __fmul_rn(kk, vv[3 % VEC]));
                *reinterpret_cast<float4*>(dst + (size_t)kd * p.Dv + col0) = n;
                o[0] = fmaf(qq, n.x, o[0]);
                o[1 % VEC] = fmaf(qq, n.y, o[1 % VEC]);
                o[2 % VEC] = fmaf(qq, n.z, o[2 % VEC]);
                o[3 % VEC] = fmaf(qq, n.w, o[3 % VEC]);
            }
        }
    } else {
        if (col0 < p.Dv) {
#pragma unroll 4
            for (int kd = rg; kd < p.Dk; kd += RG) {
                const float s = src[(size_t)kd * p.Dv + col0];
                const float n = __fadd_rn(__fmul_rn(s, decay), __fmul_rn(s_k[kd], vv[0]));
                dst[(size_t)kd * p.Dv + col0] = n;
                o[0] = fmaf(s_q[kd], n, o[0]);
            }
        }
    }

#pragma unroll
    for (int j = 0; j < VEC; ++j) s_red[rg][ct * VEC + j] = o[j];
    __syncthreads();
    if (threadIdx.x < kLinCols) {
        const int col = slice * kLinCols + threadIdx.x;
        if (col < p.Dv) {
            float sum = 0.0f;
#pragma unroll 8
            for (int r = 0; r < RG; ++r) sum += s_red[r][threadIdx.x];
            static_cast<T*>(p.out)[((size_t)b * p.Hv + h) * p.Dv + col] = from_float<T>(sum);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// The strip kernels: value_dim and key_dim multiples of four, key_dim <= 256, aligned states.
//
// A warp owns 16 value columns of one (batch, value head) state matrix: lane = (row group g = lane / 4,
// column quad c = lane % 4), and a thread keeps columns 4c .. 4c + 3 of the rows 32 i + 4 g + j (j < 4),
// 16 of 128 rows.  A load instruction of the warp takes 64 contiguous bytes of eight rows; k and q come
// from shared memory as one 128-bit word for four rows, eight groups side by side (conflict-free); and
// the read-out sum over the rows stays inside the warp: two accumulators per column (even and odd rows),
// then a reduce-scatter of four shuffles.  One-step and multi-step calls run the same arithmetic in the
// same order, so T steps in one launch are bit-identical to T launches.
// ---------------------------------------------------------------------------------------------
constexpr int kStripCols = 32;                      // value columns of a CTA
constexpr int kStripThreads = 2 * kStripCols;       // two warps of 16 columns
constexpr int kStripChunk = 4;                      // steps whose q, k, v are staged together
constexpr int kStripAhead = 3;                      // chunks on their way while one is worked on

struct LinStepsParams {
    const void* q;      // [steps][B][Hk][Dk]
    const void* k;
    const void* v;      // [steps][B][Hv][Dv]
    const float* state;
    void* out;          // [steps][B][Hv][Dv]
    float* new_state;
    const float* decay_ps;  // [steps][B][Hv] or null
    const float* beta_ps;   // [steps][B][Hv] or null
    int steps, B, Hk, Hv, Dk, Dv;
    float decay;
    float one;  // 1.0f, known at run time only
};

// four consecutive elements as fp32
template <typename T>
struct Quad { uint2 raw; };
template <>
struct Quad<float> { uint4 raw; };
template <typename T>
__device__ __forceinline__ Quad<T> load_quad(const T* p) {
    Quad<T> r;
    r.raw = *reinterpret_cast<const decltype(r.raw)*>(p);
    return r;
}
__device__ __forceinline__ float4 quad_floats(const Quad<__nv_bfloat16>& r) {
    return make_float4(__uint_as_float(r.raw.x << 16), __uint_as_float(r.raw.x & 0xffff0000u), __uint_as_float(r.raw.y << 16),
                       __uint_as_float(r.raw.y & 0xffff0000u));
}
__device__ __forceinline__ float4 quad_floats(const Quad<__half>& r) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.raw.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&r.raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 quad_floats(const Quad<float>& r) {
    return make_float4(__uint_as_float(r.raw.x), __uint_as_float(r.raw.y), __uint_as_float(r.raw.z), __uint_as_float(r.raw.w));
}

// the same where the address may be aligned to one element only
template <bool ALIGNED, typename T>
__device__ __forceinline__ float4 load_floats(const T* p) {
    if constexpr (ALIGNED) return quad_floats(load_quad(p));
    else return make_float4(to_float<T>(p[0]), to_float<T>(p[1]), to_float<T>(p[2]), to_float<T>(p[3]));
}

// Two fp32 values per instruction (each rounded on its own, as the scalar instructions round).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__host__ __device__ constexpr int strip_step_bytes(int key_dim, int elem) { return (2 * key_dim + kStripCols) * elem + 16; }

template <typename T>
__device__ __forceinline__ void cp_async_quad(T* dst, const T* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(4 * (int)sizeof(T)) : "memory");
}
template <bool ALIGNED, typename T>
__device__ __forceinline__ void stage_quad(T* dst, const T* src) {
    if constexpr (ALIGNED) {
        cp_async_quad(dst, src);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = src[i];
    }
}
__device__ __forceinline__ void cp_async4(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Sum of column sums o[0..3] over the eight row groups (lane bits 2-4).  Afterwards every lane holds the
// total of column 4 * (lane % 4) + 2 * bit4 + bit3.
__device__ __forceinline__ float reduce_columns(const float (&o)[4], int lane) {
    const bool hi = lane & 16, hj = lane & 8;
    float a = hi ? o[2] : o[0], b = hi ? o[3] : o[1];
    a += __shfl_xor_sync(kFullMask, hi ? o[0] : o[2], 16);
    b += __shfl_xor_sync(kFullMask, hi ? o[1] : o[3], 16);
    float c = hj ? b : a;
    c += __shfl_xor_sync(kFullMask, hj ? a : b, 8);
    return c + __shfl_xor_sync(kFullMask, c, 4);
}

// NQ: row quads of a thread (4: key_dim <= 128, 8: <= 256).  FULL: key_dim is exactly 32 NQ.  ALIGNED: q, k and v are aligned
// to four elements; where they are not they are read element by element, and everything else is the same (64 steps, eight
// tokens, 32 heads of 128 x 128: 59 us aligned, 71 not, 525 as 64 launches).
//
// One step: a stream through registers; all of a thread's loads are in flight before anything waits.
template <typename T, int NQ, bool FULL, bool ALIGNED>
__global__ void __launch_bounds__(kStripThreads) linear_strip_kernel(const LinParams p) {
    extern __shared__ __align__(16) float s_dyn[];  // k[Dk], q[Dk]
    const int slices = (p.Dv + kStripCols - 1) / kStripCols;
    const int slice = blockIdx.x % slices, bh = blockIdx.x / slices;
    const int b = bh / p.Hv, h = bh - b * p.Hv, hk = h / (p.Hv / p.Hk);
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2;
    const int wcol = slice * kStripCols + (tid >> 5) * 16;
    const int col0 = wcol + 4 * (lane & 3);
    const bool live = col0 < p.Dv;

    const size_t base = ((size_t)b * p.Hv + h) * p.Dk * p.Dv + col0;
    float4 st[4 * NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int kd = 32 * i + 4 * g + j;
            st[4 * i + j] = (live && (FULL || kd < p.Dk)) ? *reinterpret_cast<const float4*>(p.state + base + (size_t)kd * p.Dv) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    const size_t qk = ((size_t)b * p.Hk + hk) * p.Dk;
    float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) vv = load_floats<ALIGNED>(static_cast<const T*>(p.v) + ((size_t)b * p.Hv + h) * p.Dv + col0);
    const float decay = p.decay_ph ? p.decay_ph[(size_t)b * p.Hv + h] : p.decay;
    if (p.beta_ph) {
        const float beta = p.beta_ph[(size_t)b * p.Hv + h];
        vv.x = __fmul_rn(vv.x, beta); vv.y = __fmul_rn(vv.y, beta); vv.z = __fmul_rn(vv.z, beta); vv.w = __fmul_rn(vv.w, beta);
    }
    for (int i = tid; i < p.Dk / 2; i += kStripThreads) {  // quads of k, then of q
        const bool is_k = i < p.Dk / 4;
        const T* src = static_cast<const T*>(is_k ? p.k : p.q) + qk + 4 * (is_k ? i : i - p.Dk / 4);
        *reinterpret_cast<float4*>(s_dyn + 4 * i) = load_floats<ALIGNED>(src);
    }
    __syncthreads();
    float even[4] = {0.f, 0.f, 0.f, 0.f}, odd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        if (!live || (!FULL && 32 * i + 4 * g >= p.Dk)) continue;
        const float4 k4 = *reinterpret_cast<const float4*>(s_dyn + 32 * i + 4 * g);
        const float4 q4 = *reinterpret_cast<const float4*>(s_dyn + p.Dk + 32 * i + 4 * g);
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 n = st[4 * i + j];
            n.x = __fadd_rn(__fmul_rn(n.x, decay), __fmul_rn(kk[j], vv.x));
            n.y = __fadd_rn(__fmul_rn(n.y, decay), __fmul_rn(kk[j], vv.y));
            n.z = __fadd_rn(__fmul_rn(n.z, decay), __fmul_rn(kk[j], vv.z));
            n.w = __fadd_rn(__fmul_rn(n.w, decay), __fmul_rn(kk[j], vv.w));
            *reinterpret_cast<float4*>(p.new_state + base + (size_t)(32 * i + 4 * g + j) * p.Dv) = n;
            float(&o)[4] = (j & 1) ? odd : even;
            o[0] = fmaf(qq[j], n.x, o[0]);
            o[1] = fmaf(qq[j], n.y, o[1]);
            o[2] = fmaf(qq[j], n.z, o[2]);
            o[3] = fmaf(qq[j], n.w, o[3]);
        }
    }
    const float o[4] = {even[0] + odd[0], even[1] + odd[1], even[2] + odd[2], even[3] + odd[3]};
    const float sum = reduce_columns(o, lane);
    if (live && !(lane & 4)) {
        const int col = col0 + ((lane >> 4) << 1) + ((lane >> 3) & 1);
        static_cast<T*>(p.out)[((size_t)b * p.Hv + h) * p.Dv + col] = from_float<T>(sum);
    }
}

// Several consecutive steps in one launch, the fp32 state resident in registers for the whole call: HBM
// sees it once on the way in and once on the way out.  What bounds it then is the FP32 pipe, four
// operations per state element and step.  They are done two rows at a time (f32x2: half the instructions,
// the same pipe time); a CTA is small (32 columns: 2048 warps at eight tokens of 32 heads, 13.8 per SM);
// q, k, v travel to shared memory by asynchronous copies, kStripAhead chunks of four steps ahead, and are
// widened as they are read; and the four read-out sums of a chunk go through their shuffles together.
// Measured at 64 steps, eight tokens, 32 heads of 128 x 128: 59 us (about 29 us of it is the FP32 pipe of an average
// SM, the rest what the busiest scheduler has above the average and its other instructions); the kernel before
// it, two barriers of 256 threads and a sum through shared memory per step, took 260 us.
template <typename T, int NQ, bool FULL, bool ALIGNED>
__global__ void __launch_bounds__(kStripThreads, NQ == 4 ? 7 : 4) linear_strip_steps_kernel(const LinStepsParams p) {
    extern __shared__ __align__(16) unsigned char s_raw[];  // [kStripAhead + 1][kStripChunk][k Dk | q Dk | v kStripCols | decay, beta]
    const int slices = (p.Dv + kStripCols - 1) / kStripCols;
    const int slice = blockIdx.x % slices, bh = blockIdx.x / slices;
    const int b = bh / p.Hv, h = bh - b * p.Hv, hk = h / (p.Hv / p.Hk);
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2;
    const int wloc = (tid >> 5) * 16 + 4 * (lane & 3);  // first column of the thread inside the slice
    const int col0 = slice * kStripCols + wloc;
    const bool live = col0 < p.Dv;
    const int Dk = FULL ? 32 * NQ : p.Dk;
    const int stride = strip_step_bytes(Dk, sizeof(T));

    const size_t qk_step = (size_t)p.B * p.Hk * Dk, v_step = (size_t)p.B * p.Hv * p.Dv, g_step = (size_t)p.B * p.Hv;
    const T* q = static_cast<const T*>(p.q) + ((size_t)b * p.Hk + hk) * Dk;
    const T* k = static_cast<const T*>(p.k) + ((size_t)b * p.Hk + hk) * Dk;
    const T* v = static_cast<const T*>(p.v) + ((size_t)b * p.Hv + h) * p.Dv + slice * kStripCols;
    T* out = static_cast<T*>(p.out) + ((size_t)b * p.Hv + h) * p.Dv;
    const size_t gidx = (size_t)b * p.Hv + h;

    const size_t base = ((size_t)b * p.Hv + h) * Dk * p.Dv + col0;
    f32x2 st[2 * NQ][4];  // [row pair][column]
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int kd = 32 * i + 4 * g + 2 * j;
            float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
            if (live && (FULL || kd < Dk)) {
                s0 = *reinterpret_cast<const float4*>(p.state + base + (size_t)kd * p.Dv);
                s1 = *reinterpret_cast<const float4*>(p.state + base + (size_t)(kd + 1) * p.Dv);
            }
            st[2 * i + j][0] = pack2(s0.x, s1.x);
            st[2 * i + j][1] = pack2(s0.y, s1.y);
            st[2 * i + j][2] = pack2(s0.z, s1.z);
            st[2 * i + j][3] = pack2(s0.w, s1.w);
        }

    // Staging of a chunk: quads of the k and q rows by all threads, a quad of v by each of the first 32, the gates by
    // the first eight.
    constexpr int kRowQuads = 8 * NQ;  // quads of a padded k (or q) row
    constexpr int kVQuads = kStripCols / 4;
    auto fetch = [&](int chunk) {
        unsigned char* buf = s_raw + (chunk % (kStripAhead + 1)) * kStripChunk * stride;
        const int step0 = chunk * kStripChunk;
#pragma unroll
        for (int r = 0; r < kStripChunk * 2 * kRowQuads / kStripThreads; ++r) {
            const int idx = tid + r * kStripThreads;
            const int row = idx / kRowQuads, c = 4 * (idx % kRowQuads), step = step0 + (row >> 1);
            if (step < p.steps && (FULL || c < Dk))
                stage_quad<ALIGNED>(reinterpret_cast<T*>(buf + (row >> 1) * stride) + (row & 1) * Dk + c, ((row & 1) ? q : k) + (size_t)step * qk_step + c);
        }
        {
            const int s = tid / kVQuads, c = 4 * (tid % kVQuads), step = step0 + s;
            if (s < kStripChunk && step < p.steps && slice * kStripCols + c < p.Dv)
                stage_quad<ALIGNED>(reinterpret_cast<T*>(buf + s * stride) + 2 * Dk + c, v + (size_t)step * v_step + c);
        }
        if (tid < 2 * kStripChunk) {
            const float* gate = (tid & 1) ? p.beta_ps : p.decay_ps;
            const int step = step0 + (tid >> 1);
            if (gate && step < p.steps)
                cp_async4(reinterpret_cast<T*>(buf + (tid >> 1) * stride) + 2 * Dk + kStripCols + (tid & 1) * (4 / sizeof(T)), gate + (size_t)step * g_step + gidx);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // The products and their sum are rounded one after the other.  The assembler contracts packed multiplies and
    // adds whatever their rounding modifier says, so the sum is an FMA by a one that it cannot see through.
    const f32x2 one = pack2(p.one, p.one);

    const int nchunks = (p.steps + kStripChunk - 1) / kStripChunk;
#pragma unroll 1
    for (int c = 0; c < kStripAhead; ++c) fetch(c);  // beyond the last chunk: an empty group
    const bool hi = lane & 16, hj = lane & 8, hk4 = lane & 4;
    const int my_step = ((lane >> 4) << 1) + ((lane >> 3) & 1), col = col0 + (hk4 ? 2 : 0);
#pragma unroll 1
    for (int chunk = 0; chunk < nchunks; ++chunk) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStripAhead - 1) : "memory");
        __syncthreads();        // everybody's copies of this chunk have landed, and the last chunk's buffer is free
        fetch(chunk + kStripAhead);
        const unsigned char* buf = s_raw + (chunk % (kStripAhead + 1)) * kStripChunk * stride;
        const int step0 = chunk * kStripChunk;
        const int n = min(kStripChunk, p.steps - step0);
        float o[kStripChunk][4];
#pragma unroll
        for (int s = 0; s < kStripChunk; ++s) {
            if (s >= n) break;
            const T* row = reinterpret_cast<const T*>(buf + s * stride);
            float4 v4 = quad_floats(load_quad(row + 2 * Dk + wloc));
            const float* gates = reinterpret_cast<const float*>(row + 2 * Dk + kStripCols);
            const float d = p.decay_ps ? gates[0] : p.decay;
            if (p.beta_ps) {
                const float beta = gates[1];
                v4.x = __fmul_rn(v4.x, beta); v4.y = __fmul_rn(v4.y, beta); v4.z = __fmul_rn(v4.z, beta); v4.w = __fmul_rn(v4.w, beta);
            }
            const f32x2 dd = pack2(d, d);
            const f32x2 vv[4] = {pack2(v4.x, v4.x), pack2(v4.y, v4.y), pack2(v4.z, v4.z), pack2(v4.w, v4.w)};
            f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                if (!FULL && 32 * i + 4 * g >= Dk) continue;
                const float4 kf = quad_floats(load_quad(row + 32 * i + 4 * g)), qf = quad_floats(load_quad(row + Dk + 32 * i + 4 * g));
                const f32x2 k0 = pack2(kf.x, kf.y), k1 = pack2(kf.z, kf.w), q0 = pack2(qf.x, qf.y), q1 = pack2(qf.z, qf.w);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const f32x2 n0 = fma2(mul2(st[2 * i][c], dd), one, mul2(k0, vv[c]));
                    const f32x2 n1 = fma2(mul2(st[2 * i + 1][c], dd), one, mul2(k1, vv[c]));
                    st[2 * i][c] = n0;
                    st[2 * i + 1][c] = n1;
                    acc[c] = fma2(q1, n1, fma2(q0, n0, acc[c]));
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 e = unpack2(acc[c]);
                o[s][c] = e.x + e.y;
            }
        }
        // The sums over the row groups, all steps of the chunk together: the tree of reduce_columns (partners
        // 16, 8, 4 lanes away), spread so that a lane ends with two columns of step 2 * bit4 + bit3.
        float r1[2][4], r2[4], r3[2];
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                r1[s][c] = (hi ? o[2 + s][c] : o[s][c]) + __shfl_xor_sync(kFullMask, hi ? o[s][c] : o[2 + s][c], 16);
#pragma unroll
        for (int c = 0; c < 4; ++c) r2[c] = (hj ? r1[1][c] : r1[0][c]) + __shfl_xor_sync(kFullMask, hj ? r1[0][c] : r1[1][c], 8);
#pragma unroll
        for (int c = 0; c < 2; ++c) r3[c] = (hk4 ? r2[2 + c] : r2[c]) + __shfl_xor_sync(kFullMask, hk4 ? r2[c] : r2[2 + c], 4);
        if (live && my_step < n) {
            T* dst = out + (size_t)(step0 + my_step) * v_step + col;
            dst[0] = from_float<T>(r3[0]);
            dst[1] = from_float<T>(r3[1]);
        }
    }

#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int kd = 32 * i + 4 * g + 2 * j;
            if (live && (FULL || kd < Dk)) {
                const float2 x = unpack2(st[2 * i + j][0]), y = unpack2(st[2 * i + j][1]), z = unpack2(st[2 * i + j][2]), w = unpack2(st[2 * i + j][3]);
                *reinterpret_cast<float4*>(p.new_state + base + (size_t)kd * p.Dv) = make_float4(x.x, y.x, z.x, w.x);
                *reinterpret_cast<float4*>(p.new_state + base + (size_t)(kd + 1) * p.Dv) = make_float4(x.y, y.y, z.y, w.y);
            }
        }
}

// ---------------------------------------------------------------------------------------------
// Several steps in one launch where key_dim is not a multiple of four, which the strips need.  The partition and the arithmetic of linear_attention_kernel, in the same order, so that T steps are
// bit-identical to T of its launches; a thread keeps up to eight rows by four columns of the state in registers and the
// next step's q, k, v are fetched, element by element, while the current step is computed.  Two block-wide barriers and a
// sum through shared memory per step: four times the strips' time, but a launch per step passes the state through HBM
// each time (64 steps, eight tokens, 32 heads of 126 x 128, bf16: 200 us, as 64 launches 653).
// ---------------------------------------------------------------------------------------------
constexpr int kLinStepRows = 8;  // state rows per thread: key_dim <= 8 * 32

template <typename T>
__global__ void __launch_bounds__(kLinThreads) linear_attention_steps_kernel(const LinStepsParams p) {
    constexpr int VEC = 4;
    constexpr int CT = kLinCols / VEC;     // 8 threads across the column slice
    constexpr int RG = kLinThreads / CT;   // 32 row groups
    extern __shared__ float s_dyn[];       // q[Dk], k[Dk]
    __shared__ float s_red[RG][kLinCols + 1];
    __shared__ float s_v[kLinCols];

    const int slices = (p.Dv + kLinCols - 1) / kLinCols;
    const int slice = blockIdx.x % slices;
    const int bh = blockIdx.x / slices;
    const int h = bh % p.Hv;
    const int b = bh / p.Hv;
    const int hk = h / (p.Hv / p.Hk);
    const int tid = threadIdx.x;
    const int ct = tid % CT, rg = tid / CT;
    const int col0 = slice * kLinCols + ct * VEC;
    const bool live = col0 < p.Dv;  // Dv % 4 == 0 on this path

    float* s_q = s_dyn;
    float* s_k = s_dyn + p.Dk;
    const size_t qk_step = (size_t)p.B * p.Hk * p.Dk, v_step = (size_t)p.B * p.Hv * p.Dv, g_step = (size_t)p.B * p.Hv;
    const T* q = static_cast<const T*>(p.q) + ((size_t)b * p.Hk + hk) * p.Dk;
    const T* k = static_cast<const T*>(p.k) + ((size_t)b * p.Hk + hk) * p.Dk;
    const T* v = static_cast<const T*>(p.v) + ((size_t)b * p.Hv + h) * p.Dv + slice * kLinCols;
    T* out = static_cast<T*>(p.out) + ((size_t)b * p.Hv + h) * p.Dv + slice * kLinCols;
    const size_t gidx = (size_t)b * p.Hv + h;

    // the state slice of this thread: rows rg, rg + 32, ... x 4 columns
    const size_t base = ((size_t)b * p.Hv + h) * p.Dk * p.Dv;
    float4 st[kLinStepRows];
#pragma unroll
    for (int r = 0; r < kLinStepRows; ++r) {
        const int kd = rg + r * RG;
        st[r] = (live && kd < p.Dk) ? *reinterpret_cast<const float4*>(p.state + base + (size_t)kd * p.Dv + col0)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }

    // software pipeline: thread i carries element i (and i + 256) of the next step's q and k, and
    // the first 32 threads the next step's v slice
    auto fetch = [&](int step, float (&nq)[2], float (&nk)[2], float& nv) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = tid + j * kLinThreads;
            nq[j] = (i < p.Dk) ? to_float<T>(q[(size_t)step * qk_step + i]) : 0.0f;
            nk[j] = (i < p.Dk) ? to_float<T>(k[(size_t)step * qk_step + i]) : 0.0f;
        }
        nv = (tid < kLinCols && slice * kLinCols + tid < p.Dv) ? to_float<T>(v[(size_t)step * v_step + tid]) : 0.0f;
    };
    float nq[2], nk[2], nv;
    fetch(0, nq, nk, nv);

    for (int step = 0; step < p.steps; ++step) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = tid + j * kLinThreads;
            if (i < p.Dk) { s_q[i] = nq[j]; s_k[i] = nk[j]; }
        }
        if (tid < kLinCols) s_v[tid] = nv;
        const float decay = p.decay_ps ? p.decay_ps[(size_t)step * g_step + gidx] : p.decay;
        const float beta = p.beta_ps ? p.beta_ps[(size_t)step * g_step + gidx] : 1.0f;
        __syncthreads();
        if (step + 1 < p.steps) fetch(step + 1, nq, nk, nv);

        float vv[VEC], o[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const float raw = s_v[ct * VEC + j];
            vv[j] = p.beta_ps ? __fmul_rn(raw, beta) : raw;
            o[j] = 0.0f;
        }
        if (live) {
#pragma unroll
            for (int r = 0; r < kLinStepRows; ++r) {
                const int kd = rg + r * RG;
                if (kd < p.Dk) {
                    const float kk = s_k[kd], qq = s_q[kd];
                    float4 n;
                    n.x = __fadd_rn(__fmul_rn(st[r].x, decay), __fmul_rn(kk, vv[0]));
                    n.y = __fadd_rn(__fmul_rn(st[r].y, decay), __fmul_rn(kk, vv[1]));
                    n.z = __fadd_rn(__fmul_rn(st[r].z, decay), __fmul_rn(kk, vv[2]));
                    n.w = __fadd_rn(__fmul_rn(st[r].w, decay), __fmul_rn(kk, vv[3]));
                    st[r] = n;
                    o[0] = fmaf(qq, n.x, o[0]);
                    o[1] = fmaf(qq, n.y, o[1]);
                    o[2] = fmaf(qq, n.z, o[2]);
                    o[3] = fmaf(qq, n.w, o[3]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < VEC; ++j) s_red[rg][ct * VEC + j] = o[j];
        __syncthreads();
        if (tid < kLinCols && slice * kLinCols + tid < p.Dv) {
            float sum = 0.0f;
#pragma unroll 8
            for (int r = 0; r < RG; ++r) sum += s_red[r][tid];
            out[(size_t)step * v_step + tid] = from_float<T>(sum);
        }
        // the next iteration's writes to s_q / s_k / s_v happen after everyone has passed the barrier
        // above; its writes to s_red come after its own first barrier, i.e. after the sums were read
    }

#pragma unroll
    for (int r = 0; r < kLinStepRows; ++r) {
        const int kd = rg + r * RG;
        if (live && kd < p.Dk) *reinterpret_cast<float4*>(p.new_state + base + (size_t)kd * p.Dv + col0) = st[r];
    }
}

// Whether the strip kernels take a call.  Both the one-step and the multi-step entry point ask this, and neither the answer
// nor the order of the sums depends on the alignment of q, k and v, so that their results agree bit for bit.
bool strip_fits(int key_dim, int value_dim, const float* state, const float* new_state) {
    const uintptr_t st = reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(new_state);
    return value_dim % 4 == 0 && key_dim % 4 == 0 && key_dim <= 256 && (st & 15u) == 0;
}
template <typename T>
bool quads_aligned(const void* q, const void* k, const void* v) {
    return ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & (4 * sizeof(T) - 1)) == 0;
}

template <typename T>
int launch_linear(const LinParams& p, cudaStream_t stream) {
    const int slices = (p.Dv + kLinCols - 1) / kLinCols;
    const long long ctas = (long long)p.B * p.Hv * slices;
    if (ctas > 0x7fffffffLL) MK36_FAIL(MK36_ERR_UNSUPPORTED, "linear_attention_decode: too many (batch, head) pairs");
    const size_t smem = (size_t)2 * p.Dk * sizeof(float);
    if (smem > 40 * 1024) MK36_FAIL(MK36_ERR_UNSUPPORTED, "linear_attention_decode: key_dim %d is too large", p.Dk);
    if (strip_fits(p.Dk, p.Dv, p.state, p.new_state)) {
        const bool aligned = quads_aligned<T>(p.q, p.k, p.v);
        if (!aligned && p.Dk <= 128) linear_strip_kernel<T, 4, false, false><<<(unsigned)ctas, kStripThreads, smem, stream>>>(p);
        else if (!aligned) linear_strip_kernel<T, 8, false, false><<<(unsigned)ctas, kStripThreads, smem, stream>>>(p);
        else if (p.Dk == 128) linear_strip_kernel<T, 4, true, true><<<(unsigned)ctas, kStripThreads, smem, stream>>>(p);
        else if (p.Dk < 128) linear_strip_kernel<T, 4, false, true><<<(unsigned)ctas, kStripThreads, smem, stream>>>(p);
        else linear_strip_kernel<T, 8, false, true><<<(unsigned)ctas, kStripThreads, smem, stream>>>(p);
        MK36_CUDA_OK(cudaGetLastError());
        return MK36_OK;
    }
    // key_dim above 256, a dimension that is not a multiple of four, or an unaligned state
    const bool vec = (p.Dv % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.state) & 15u) == 0) &&
                     ((reinterpret_cast<uintptr_t>(p.new_state) & 15u) == 0);
    if (vec) linear_attention_kernel<T, 4><<<(unsigned)ctas, kLinThreads, smem, stream>>>(p);
    else linear_attention_kernel<T, 1><<<(unsigned)ctas, kLinThreads, smem, stream>>>(p);
    MK36_CUDA_OK(cudaGetLastError());
    return MK36_OK;
}

template <typename T>
void launch_steps(const LinStepsParams& p, bool strip, unsigned ctas, cudaStream_t stream) {
    if (!strip) {
        linear_attention_steps_kernel<T><<<ctas, kLinThreads, (size_t)2 * p.Dk * sizeof(float), stream>>>(p);
        return;
    }
    const size_t smem = (size_t)(kStripAhead + 1) * kStripChunk * strip_step_bytes(p.Dk, sizeof(T));  // at most 35 KB
    const bool aligned = quads_aligned<T>(p.q, p.k, p.v);
    if (!aligned && p.Dk <= 128) linear_strip_steps_kernel<T, 4, false, false><<<ctas, kStripThreads, smem, stream>>>(p);
    else if (!aligned) linear_strip_steps_kernel<T, 8, false, false><<<ctas, kStripThreads, smem, stream>>>(p);
    else if (p.Dk == 128) linear_strip_steps_kernel<T, 4, true, true><<<ctas, kStripThreads, smem, stream>>>(p);
    else if (p.Dk < 128) linear_strip_steps_kernel<T, 4, false, true><<<ctas, kStripThreads, smem, stream>>>(p);
    else linear_strip_steps_kernel<T, 8, false, true><<<ctas, kStripThreads, smem, stream>>>(p);
}

}  // namespace mk36

using namespace mk36;

extern "C" int mk36_linear_attention_decode(const mk36_linear_attention_args* a, void* stream) {
    if (!a) MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode: args is NULL");
    if (!a->q || !a->k || !a->v || !a->state || !a->out || !a->new_state)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode: NULL tensor pointer");
    if (a->batch <= 0 || a->key_heads <= 0 || a->value_heads <= 0 || a->key_dim <= 0 || a->value_dim <= 0)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode: sizes must be positive");
    if (a->value_heads % a->key_heads != 0)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode: value_heads must be a multiple of key_heads");
    if (!current_device_info()) return MK36_ERR_LAUNCH;
    LinParams p;
    p.q = a->q;
    p.k = a->k;
    p.v = a->v;
    p.state = a->state;
    p.out = a->out;
    p.new_state = a->new_state;
    p.decay_ph = a->decay_per_head;
    p.beta_ph = a->beta_per_head;
    p.B = a->batch;
    p.Hk = a->key_heads;
    p.Hv = a->value_heads;
    p.Dk = a->key_dim;
    p.Dv = a->value_dim;
    p.decay = a->decay;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (a->dtype) {
        case MK36_BF16: return launch_linear<__nv_bfloat16>(p, s);
        case MK36_F16: return launch_linear<__half>(p, s);
        case MK36_F32: return launch_linear<float>(p, s);
        default: MK36_FAIL(MK36_ERR_UNSUPPORTED, "linear_attention_decode: unsupported dtype %d", a->dtype);
    }
}

// Several steps in one call: the strips, else the state in registers all the same.  What remains (value_dim not a multiple
// of four, key_dim above 256, an unaligned state) runs the single-step kernel once per step on the same stream, with the
// same results.
extern "C" int mk36_linear_attention_decode_steps(const mk36_linear_attention_steps_args* a, void* stream) {
    if (!a) MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode_steps: args is NULL");
    if (!a->q || !a->k || !a->v || !a->state || !a->out || !a->new_state)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode_steps: NULL tensor pointer");
    if (a->steps <= 0 || a->batch <= 0 || a->key_heads <= 0 || a->value_heads <= 0 || a->key_dim <= 0 || a->value_dim <= 0)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode_steps: sizes must be positive");
    if (a->value_heads % a->key_heads != 0)
        MK36_FAIL(MK36_ERR_INVALID_ARG, "linear_attention_decode_steps: value_heads must be a multiple of key_heads");
    if (a->dtype != MK36_BF16 && a->dtype != MK36_F16 && a->dtype != MK36_F32)
        MK36_FAIL(MK36_ERR_UNSUPPORTED, "linear_attention_decode_steps: unsupported dtype %d", a->dtype);
    if (!current_device_info()) return MK36_ERR_LAUNCH;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool strip = strip_fits(a->key_dim, a->value_dim, a->state, a->new_state);
    const bool resident = a->value_dim % 4 == 0 && a->key_dim <= kLinStepRows * 32 &&
                          ((reinterpret_cast<uintptr_t>(a->state) | reinterpret_cast<uintptr_t>(a->new_state)) & 15u) == 0;
    const size_t es = a->dtype == MK36_F32 ? 4 : 2;
    if (!resident) {
        const size_t qk = (size_t)a->batch * a->key_heads * a->key_dim * es, vb = (size_t)a->batch * a->value_heads * a->value_dim * es;
        const size_t gs = (size_t)a->batch * a->value_heads;
        for (int t = 0; t < a->steps; ++t) {
            mk36_linear_attention_args one{};
            one.q = static_cast<const unsigned char*>(a->q) + t * qk;
            one.k = static_cast<const unsigned char*>(a->k) + t * qk;
            one.v = static_cast<const unsigned char*>(a->v) + t * vb;
            one.state = (t == 0) ? a->state : a->new_state;  // in place from the second step on
            one.out = static_cast<unsigned char*>(a->out) + t * vb;
            one.new_state = a->new_state;
            one.decay_per_head = a->decay_per_step ? a->decay_per_step + t * gs : nullptr;
            one.beta_per_head = a->beta_per_step ? a->beta_per_step + t * gs : nullptr;
            one.dtype = a->dtype;
            one.batch = a->batch;
            one.key_heads = a->key_heads;
            one.value_heads = a->value_heads;
            one.key_dim = a->key_dim;
            one.value_dim = a->value_dim;
            one.decay = a->decay;
            const int rc = mk36_linear_attention_decode(&one, stream);
            if (rc != MK36_OK) return rc;
        }
        return MK36_OK;
    }
    LinStepsParams p;
    p.q = a->q; p.k = a->k; p.v = a->v;
    p.state = a->state; p.out = a->out; p.new_state = a->new_state;
    p.decay_ps = a->decay_per_step; p.beta_ps = a->beta_per_step;
    p.steps = a->steps; p.B = a->batch; p.Hk = a->key_heads; p.Hv = a->value_heads; p.Dk = a->key_dim; p.Dv = a->value_dim;
    p.decay = a->decay;
    p.one = 1.0f;
    const long long ctas = (long long)p.B * p.Hv * ((p.Dv + kStripCols - 1) / kStripCols);
    if (ctas > 0x7fffffffLL) MK36_FAIL(MK36_ERR_UNSUPPORTED, "linear_attention_decode_steps: too many (batch, head) pairs");
    switch (a->dtype) {
        case MK36_BF16: launch_steps<__nv_bfloat16>(p, strip, (unsigned)ctas, s); break;
        case MK36_F16: launch_steps<__half>(p, strip, (unsigned)ctas, s); break;
        default: launch_steps<float>(p, strip, (unsigned)ctas, s); break;
    }
    MK36_CUDA_OK(cudaGetLastError());
    return MK36_OK;
}
