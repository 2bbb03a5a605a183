// MoE decode for launches of up to 32 tokens on sm_100a (bf16, aligned shapes): every distinct expert's
// weights are read once for all tokens of the launch.  Same results as the general kernel in
// moe_decode.cu (reference semantics: mega_kernel_qwen36/reference.py:16-62).
//
// What bounds it: the weight stream.  32 tokens with eight experts each meet about 163 distinct experts
// of 256 (1.03 GB at hidden 2048, width 512); four launches of eight tokens read 58 each, 40 % more, and
// pay their latencies four times.  An expert has one to five tokens, which are columns of
// mma.sync.m16n8k16, so the arithmetic does not grow with them.  As in dense_ffn_mma.cu the weights go
// from global memory into fragments, eight 32-wide slices ahead (96 KB in flight per SM), which leaves
// the shared memory to the 32 normalised tokens.  A lane loads 32 bytes at once, so that a fragment load
// covers whole 128-byte lines: 16-byte loads took 204 against 188 us.  Twelve warps: 16 with 128 registers
// took 193, 8 with twice the slices in flight 202.
//
// Hidden 2048, 256 experts of width 512, top 8, bf16, 32 tokens: 315 us as four launches of the batch
// kernel, 205 here (1.03 GB: 5.0 TB/s).
//
// Sums: the tensor core cuts off where an fp32 addition rounds.  As one chain of MMAs over a whole sum the
// fp32 output was eight times as far from the 64-bit sum as the batch kernel's, which rounds every addition
// (relative error 1.25e-6 against 1.6e-7).  So a 32-wide slice is a chain of its own from zero, slices are
// added up in fp32, and what is done a few times per value (the four shares of a gate/up tile, silu(g) * u
// behind the exponential, the slots of a token) in fp64: 1.6e-7 as well, at 3 % (32 tokens 198 -> 205 us).
// Taken back: pieces of eight products (no closer, 8 % slower); even and odd accumulators or fp64 in the down
// sums too (1.55e-7 and 1.45e-7, 217 and 219 us).
//
//   phase 0   every CTA normalises all tokens into shared memory and dots them with its one or two
//             router rows (fp32 FMA, as in the other kernels; the sum of squares of a token is one warp's
//             chain here, so that a near tie of two logits may still fall differently)     | arrive 1
//   phase A'  the shared expert's gate/up units (they need no routing)                   | wait 1
//   select    every CTA: top-k and soft-max per token, list of entries = (expert, up to eight of its
//             tokens); an expert with more tokens has several entries, which share its weights in L2
//   phase A   unit = 8 gate + 8 up rows of an entry, by four warps that split the hidden length; they
//             add up in shared memory; silu(g) * u, an fp32 value, is stored as three bf16 terms whose
//             sum is that value exactly                                                 | barrier 2
//   phase C   the CTA's output rows (at most 16) of every entry's down matrix, an entry per warp; three
//             MMAs per slice pair, one per term, so nothing of the activation is lost
//   combine   in slot order, residual, one rounding
#include "mk36_mma.cuh"
#include "mk36_moe_stream.cuh"

namespace mk36 {

constexpr int kWdWarps = 12;                          // 168 registers per thread: the slices in flight live there
constexpr int kWdThreads = kWdWarps * 32;
constexpr int kWdQuadWarps = 4;                       // warps that share a gate/up unit
constexpr int kWdQuads = kWdWarps / kWdQuadWarps;
constexpr int kWdMaxTokens = 32;
constexpr int kWdCols = 8;                            // tokens of an entry: columns of the tile
constexpr int kWdSlots = 8;                           // pair (token b, slot r) has index b * 8 + r
constexpr int kWdPairs = kWdMaxTokens * kWdSlots;     // the shared expert's pair of token b is kWdPairs + b
constexpr int kWdMaxEntries = kWdPairs + kWdMaxTokens / kWdCols;
constexpr int kWdAhead = 8;                           // 32-wide slices in flight per warp
constexpr int kWdDownAhead = 8;                       // the same in phase C, where the activations' terms need registers too
constexpr int kWdPieces = 8;                          // 16-byte pieces of a token per lane: hidden <= 2048
constexpr int kWdRouterRows = 2;                      // router rows per CTA
constexpr int kWdTokensPerWarp = (kWdMaxTokens + kWdWarps - 1) / kWdWarps;
constexpr int kWdPad = 8;                             // elements: rows 16 bytes apart modulo 128, so that fragment loads meet all banks

struct MoeWideParams {
    const __nv_bfloat16* x;
    const __nv_bfloat16* norm_w;
    const __nv_bfloat16* router_w;
    const __nv_bfloat16* egate;
    const __nv_bfloat16* eup;
    const __nv_bfloat16* edown;
    const __nv_bfloat16* sgate;
    const __nv_bfloat16* sup;
    const __nv_bfloat16* sdown;
    __nv_bfloat16* out;
    long long* indices;
    float* route_w;
    float* partial_out;
    Control* ctl;
    float* logits;         // [token][E]
    __nv_bfloat16* act;    // [pair][3][I]: the three terms of silu(gate) * up
    __nv_bfloat16* sact;   // [token][3][Is]
    int ntok, H, E, K, I, Is;
    int expert_base, local_experts, add_residual;
    float eps;
    int hr_max;
    int off_part, off_row, off_norm, off_slot, off_emask, off_ent_e, off_ent_m, off_ent_tok, off_ent_pair, off_pair_e, off_pair_w, off_x;
    FastDiv fd_tiles, fd_stiles;  // gate/up tiles of a routed / the shared expert
};

// v = hi + mid + lo exactly: truncation leaves 8 of the 24 significand bits per term.  Infinities and NaN stay in hi.
__device__ __forceinline__ void split3(float v, __nv_bfloat16& hi, __nv_bfloat16& mid, __nv_bfloat16& lo) {
    const float h = __uint_as_float(__float_as_uint(v) & 0xffff0000u);
    const float r = v - h;
    const float m = __uint_as_float(__float_as_uint(r) & 0xffff0000u);
    const bool finite = fabsf(v) < INFINITY;
    hi = __float2bfloat16_rn(finite ? h : v);
    mid = __float2bfloat16_rn(finite ? m : 0.0f);
    lo = __float2bfloat16_rn(finite ? r - m : 0.0f);
}

// silu(g) * u with one rounding behind the exponential
__device__ __forceinline__ float swiglu_exact(float g, float u) { return (float)((double)g * u / (1.0 + expf(-g))); }

// Gate/up units [first, end) in steps of `step`, tile units of the entries from `entry0`, by the four warps of a quad.
struct WideGateUp {
    const __nv_bfloat16* gate;
    const __nv_bfloat16* up;
    __nv_bfloat16* act;       // of pair `pair0`
    int pair0, I, entry0, expert_base;
    FastDiv tiles;
};

__device__ __forceinline__ void wide_gate_up(const WideGateUp w, int first, int end, int step, int H, const __nv_bfloat16* xs, const int* ent_e,
                                          const unsigned char* ent_tok, const short* ent_pair, float4* part, int quad, int kpart, int lane) {
    using T = __nv_bfloat16;
    const int g = lane >> 2, t = lane & 3;
    const int S = H / (32 * kWdQuadWarps);  // slices of this warp's quarter of the hidden length
    const int R = S / kWdAhead;             // whole rounds of slices
    const int x_stride = H + kWdPad;
    const size_t koff = (size_t)kpart * S * 32 + 16 * t;

    auto row_offset = [&](int u, int& entry) -> size_t {
        int tile;
        fdivmod(u, w.tiles, entry, tile);
        entry += w.entry0;
        return ((size_t)(ent_e[entry] - w.expert_base) * w.I + (size_t)tile * 8 + g) * H + koff;
    };
    if (first >= end) return;
    int entry, next_entry = 0;
    size_t off = row_offset(first, entry);
    uint4 qa[kWdAhead], qb[kWdAhead];
#pragma unroll
    for (int j = 0; j < kWdAhead; j += 2) {
        ld_stream_2u4(w.gate + off + 32 * j, qa[j], qa[j + 1]);
        ld_stream_2u4(w.up + off + 32 * j, qb[j], qb[j + 1]);
    }
    int parity = 0, turn = 0;
#pragma unroll 1
    for (int u = first; u < end; u += step) {
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
        float d2[4] = {0.f, 0.f, 0.f, 0.f}, d3[4] = {0.f, 0.f, 0.f, 0.f};
        const T* bcol = xs + (size_t)ent_tok[entry * kWdCols + g] * x_stride + koff;
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            const bool same = r + 1 < R;
            const bool more = same || u + step < end;
            if (same) off += 32 * kWdAhead;
            else if (more) off = row_offset(u + step, next_entry);
            const T* na = w.gate + off;
            const T* nb = w.up + off;
#pragma unroll
            for (int j = 0; j < kWdAhead; j += 2) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_slice32<T>(s0, s1, qa[j + q], qb[j + q], lds128(bcol + 32 * j + 8 * q));
                    add_tile(q ? d2 : d0, s0);
                    add_tile(q ? d3 : d1, s1);
                }
                if (more) {
                    ld_stream_2u4(na + 32 * j, qa[j], qa[j + 1]);
                    ld_stream_2u4(nb + 32 * j, qb[j], qb[j + 1]);
                }
            }
            bcol += 32 * kWdAhead;
        }
        add_tile(d0, d2);
        add_tile(d1, d3);
        // the quad's four shares of the tile; the warps take turns at finishing one.  Two buffers: a warp that
        // reads this one has left it before it arrives at the next unit's barrier.
        float4* mine = part + (size_t)((parity * kWdQuads + quad) * kWdQuadWarps) * 32;
        mine[kpart * 32 + lane] = make_float4(d0[0] + d1[0], d0[1] + d1[1], d0[2] + d1[2], d0[3] + d1[3]);
        named_barrier(1 + quad, kWdQuadWarps * 32);
        if (kpart == turn) {
            const float4 v0 = mine[lane];
            double vx = v0.x, vy = v0.y, vz = v0.z, vw = v0.w;
#pragma unroll
            for (int q = 1; q < kWdQuadWarps; ++q) {
                const float4 o = mine[q * 32 + lane];
                vx += o.x; vy += o.y; vz += o.z; vw += o.w;
            }
            const float4 v = make_float4((float)vx, (float)vy, (float)vz, (float)vw);
            int e_unused, tile;
            fdivmod(u, w.tiles, e_unused, tile);
            const int ch = tile * 8 + g;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int pair = ent_pair[entry * kWdCols + 2 * t + c];
                if (pair >= 0) {
                    T hi, mid, lo;
                    split3(c == 0 ? swiglu_exact(v.x, v.z) : swiglu_exact(v.y, v.w), hi, mid, lo);
                    T* dst = w.act + (size_t)(pair - w.pair0) * 3 * w.I + ch;
                    dst[0] = hi;
                    dst[w.I] = mid;
                    dst[2 * w.I] = lo;
                }
            }
        }
        parity ^= 1;
        turn = (turn + 1) & (kWdQuadWarps - 1);
        entry = next_entry;
    }
}

// The elements of a warp's down products that came out as NaN, once more from the activations' values instead of their
// terms: an infinite weight times a term that is zero is a NaN where the activation itself gives an infinity.
static __device__ __noinline__ void wide_down_again(const MoeWideParams& p, float* part_out, const int* ent_e, const short* ent_pair, int entries, int nsh,
                                                    int h0, int hr, int warp, int lane) {
    __syncwarp();
    for (int i = warp; i < entries; i += kWdWarps) {
        const int len = i < nsh ? p.Is : p.I;
        const __nv_bfloat16* rows = (i < nsh ? p.sdown : p.edown + (size_t)(ent_e[i] - p.expert_base) * p.H * p.I) + (size_t)h0 * len;
        for (int c = 0; c < kWdCols; ++c) {
            const int pair = ent_pair[i * kWdCols + c];
            if (pair < 0) continue;
            const __nv_bfloat16* act = pair >= kWdPairs ? p.sact + (size_t)(pair - kWdPairs) * 3 * p.Is : p.act + (size_t)pair * 3 * p.I;
            for (int r = 0; r < hr; ++r) {
                float* at = part_out + pair * p.hr_max + r;
                if (!isnan(*at)) continue;  // the same for the whole warp
                float sum = 0.0f;
                for (int k = lane; k < len; k += 32) {
                    const float a = (to_float(__ldcg(act + k)) + to_float(__ldcg(act + len + k))) + to_float(__ldcg(act + 2 * len + k));
                    sum = fmaf(a, to_float(rows[(size_t)r * len + k]), sum);
                }
                sum = warp_sum(sum);
                if (lane == 0) *at = sum;
            }
        }
    }
}

__global__ void __launch_bounds__(kWdThreads, 1) moe_decode_wide_kernel(const __grid_constant__ MoeWideParams p) {
    using T = __nv_bfloat16;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_flag;
    __shared__ int s_entries;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cta = blockIdx.x, ncta = gridDim.x;
    const int quad = warp / kWdQuadWarps, kpart = warp % kWdQuadWarps;
    const int H = p.H;
    const int x_stride = H + kWdPad;

    T* xs = reinterpret_cast<T*>(smem + p.off_x);                // [token][H + pad]
    float* part_out = reinterpret_cast<float*>(smem + p.off_x);  // phase C, over the tokens: [pair][hr_max]
    float4* part = reinterpret_cast<float4*>(smem + p.off_part);
    T* s_row = reinterpret_cast<T*>(smem + p.off_row);
    T* s_norm = reinterpret_cast<T*>(smem + p.off_norm);
    unsigned char* s_slot = smem + p.off_slot;                   // [expert][token]: the slot in which the token chose it
    unsigned* s_emask = reinterpret_cast<unsigned*>(smem + p.off_emask);  // per expert, the tokens that chose it
    int* ent_e = reinterpret_cast<int*>(smem + p.off_ent_e);
    unsigned* ent_m = reinterpret_cast<unsigned*>(smem + p.off_ent_m);
    unsigned char* ent_tok = smem + p.off_ent_tok;               // [entry][column]; a column without a token repeats token 0
    short* ent_pair = reinterpret_cast<short*>(smem + p.off_ent_pair);  // [entry][column]; -1: no token
    int* s_pair_e = reinterpret_cast<int*>(smem + p.off_pair_e);
    float* s_pair_w = reinterpret_cast<float*>(smem + p.off_pair_w);

    const int h0 = (int)(((long long)H * cta) / ncta), h1 = (int)(((long long)H * (cta + 1)) / ncta);
    const int hr = h1 - h0;
    const bool tracer = (cta == 0 && tid == 0);
    if (tracer) trace_stamp(p.ctl, 0);

    // ---- phase 0: RMSNorm and router logits; warp w has tokens w, w + 12, w + 24, lane l pieces l, l + 32, ... ----
    {
        const int npieces = H >> 3;
        const int r0 = (int)(((long long)p.E * cta) / ncta), r1 = (int)(((long long)p.E * (cta + 1)) / ncta);
        uint4 xv[kWdTokensPerWarp][kWdPieces];
#pragma unroll
        for (int k = 0; k < kWdTokensPerWarp; ++k) {
            const int b = warp + k * kWdWarps;
#pragma unroll
            for (int i = 0; i < kWdPieces; ++i) {
                const int piece = lane + 32 * i;
                xv[k][i] = make_uint4(0, 0, 0, 0);
                if (b < p.ntok && piece < npieces) xv[k][i] = *reinterpret_cast<const uint4*>(p.x + (size_t)b * H + 8 * piece);
            }
        }
        for (int i = tid; i < kWdRouterRows * npieces; i += kWdThreads) {
            const int row = r0 + i / npieces;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < r1) v = ld_stream_u4(p.router_w + (size_t)r0 * H + 8 * (size_t)i);
            *reinterpret_cast<uint4*>(s_row + 8 * i) = v;
        }
        for (int i = tid; i < npieces; i += kWdThreads)
            *reinterpret_cast<uint4*>(s_norm + 8 * i) = *reinterpret_cast<const uint4*>(p.norm_w + 8 * i);
        for (int e = tid; e < p.E; e += kWdThreads) s_emask[e] = 0u;
        // the shared expert's entries come first: eight tokens each
        const int nsh = (p.Is > 0) ? (p.ntok + kWdCols - 1) / kWdCols : 0;
        if (tid < nsh * kWdCols) {
            ent_e[tid / kWdCols] = 0;
            ent_tok[tid] = (unsigned char)(tid < p.ntok ? tid : 0);
            ent_pair[tid] = (short)(tid < p.ntok ? kWdPairs + tid : -1);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kWdTokensPerWarp; ++k) {
            const int b = warp + k * kWdWarps;
            if (b < p.ntok) {
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < kWdPieces; ++i) {
                    float f[8];
                    st_unpack<T>(xv[k][i], f);
#pragma unroll
                    for (int q = 0; q < 8; ++q) ss = fmaf(f[q], f[q], ss);
                }
                ss = warp_sum(ss);
                const float rstd = 1.0f / sqrtf(ss / (float)H + p.eps);
                float acc[kWdRouterRows] = {0.0f, 0.0f};
#pragma unroll
                for (int i = 0; i < kWdPieces; ++i) {
                    const int piece = lane + 32 * i;
                    if (piece < npieces) {
                        float f[8], n[8];
                        st_unpack<T>(xv[k][i], f);
                        st_unpack<T>(lds128(s_norm + 8 * piece), n);
                        T o[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            o[q] = from_float<T>(__fmul_rn(__fmul_rn(f[q], rstd), n[q]));
                            f[q] = to_float<T>(o[q]);
                        }
                        *reinterpret_cast<uint4*>(xs + (size_t)b * x_stride + 8 * piece) = *reinterpret_cast<const uint4*>(o);
#pragma unroll
                        for (int r = 0; r < kWdRouterRows; ++r) {
                            float w[8];
                            st_unpack<T>(lds128(s_row + (size_t)r * H + 8 * piece), w);
#pragma unroll
                            for (int q = 0; q < 8; ++q) acc[r] = fmaf(w[q], f[q], acc[r]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < kWdRouterRows; ++r) {
                    acc[r] = warp_sum(acc[r]);
                    if (lane == 0 && r0 + r < r1) p.logits[(size_t)b * p.E + r0 + r] = acc[r];
                }
            }
        }
    }
    const int nsh = (p.Is > 0) ? (p.ntok + kWdCols - 1) / kWdCols : 0;
    __syncthreads();
    unsigned target = 0;
    if (tid == 0) target = barrier_arrive(p.ctl, ncta, 0);
    if (tracer) trace_stamp(p.ctl, 1);

    // unit u goes to quad u mod (CTAs * quads), neighbouring units to different CTAs
    const int first_unit = quad * ncta + cta, unit_step = kWdQuads * ncta;
    // ---- phase A': the shared expert ----
    if (p.Is > 0) {
        WideGateUp w;
        w.gate = p.sgate; w.up = p.sup; w.act = p.sact;
        w.pair0 = kWdPairs; w.I = p.Is; w.entry0 = 0; w.expert_base = 0;
        w.tiles = p.fd_stiles;
        wide_gate_up(w, first_unit, nsh * (int)p.fd_stiles.d, unit_step, H, xs, ent_e, ent_tok, ent_pair, part, quad, kpart, lane);
    }
    if (tracer) trace_stamp(p.ctl, 2);
    if (tid == 0) s_flag = barrier_wait(p.ctl, target, kStatusMoeBarrier1) ? 1 : 0;
    __syncthreads();
    if (!s_flag) return;
    if (tracer) trace_stamp(p.ctl, 3);

    // ---- select: warp w routes the same tokens ----
#pragma unroll 1
    for (int b = warp; b < p.ntok; b += kWdWarps) {
        unsigned k8[kStTopkPerLane];
#pragma unroll
        for (int j = 0; j < kStTopkPerLane; ++j) {
            const int e = lane + 32 * j;
            k8[j] = (e < p.E) ? topk_key(__float_as_uint(__ldcg(p.logits + (size_t)b * p.E + e))) : 0u;
        }
        topk_select(k8, p.K, lane, [&](int r, int e, float logit) {
            s_pair_e[b * kWdSlots + r] = e;
            s_pair_w[b * kWdSlots + r] = logit;
            if (e >= p.expert_base && e < p.expert_base + p.local_experts) {
                s_slot[e * kWdMaxTokens + b] = (unsigned char)r;
                atomicOr(&s_emask[e], 1u << b);
            }
        });
        __syncwarp();
        const float top = s_pair_w[b * kWdSlots];
        const float ev = (lane < p.K) ? expf(s_pair_w[b * kWdSlots + lane] - top) : 0.0f;
        const float denom = warp_sum(ev);
        __syncwarp();
        if (lane < p.K) {
            const float wgt = ev / denom;
            s_pair_w[b * kWdSlots + lane] = wgt;
            if (cta == 0) {
                p.indices[(size_t)b * p.K + lane] = (long long)s_pair_e[b * kWdSlots + lane];
                p.route_w[(size_t)b * p.K + lane] = wgt;
            }
        }
    }
    __syncthreads();
    // entries in expert order; lane l of warp 0 scans experts 8 l .. 8 l + 7
    if (warp == 0) {
        unsigned mm[kStTopkPerLane];
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < kStTopkPerLane; ++j) {
            const int e = lane * kStTopkPerLane + j;
            mm[j] = (e < p.E) ? s_emask[e] : 0u;
            cnt += (__popc(mm[j]) + kWdCols - 1) / kWdCols;
        }
        int incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(kFullMask, incl, off);
            if (lane >= off) incl += v;
        }
        int pos = nsh + incl - cnt;
#pragma unroll
        for (int j = 0; j < kStTopkPerLane; ++j) {
            unsigned m = mm[j];
            while (m) {
                unsigned rest = m;
                for (int q = 0; q < kWdCols && rest; ++q) rest &= rest - 1u;
                ent_e[pos] = lane * kStTopkPerLane + j;
                ent_m[pos] = m & ~rest;
                ++pos;
                m = rest;
            }
        }
        if (lane == 31) s_entries = nsh + incl;
    }
    __syncthreads();
    const int entries = s_entries;
    for (int i = nsh * kWdCols + tid; i < entries * kWdCols; i += kWdThreads) {
        const int entry = i / kWdCols;
        unsigned m = ent_m[entry];
        for (int q = 0; q < i % kWdCols; ++q) m &= m - 1u;
        const int b = __ffs((int)m) - 1;
        ent_tok[i] = (unsigned char)(b < 0 ? 0 : b);
        ent_pair[i] = (short)(b < 0 ? -1 : b * kWdSlots + s_slot[ent_e[entry] * kWdMaxTokens + b]);
    }
    __syncthreads();
    if (tracer) trace_stamp(p.ctl, 4);

    // ---- phase A: the routed experts ----
    {
        WideGateUp w;
        w.gate = p.egate; w.up = p.eup; w.act = p.act;
        w.pair0 = 0; w.I = p.I; w.entry0 = nsh; w.expert_base = p.expert_base;
        w.tiles = p.fd_tiles;
        wide_gate_up(w, first_unit, (entries - nsh) * (int)p.fd_tiles.d, unit_step, H, xs, ent_e, ent_tok, ent_pair, part, quad, kpart, lane);
    }
    if (tracer) trace_stamp(p.ctl, 5);

    // ---- phase C: this CTA's down rows; entry i goes to warp i mod 12.  The first weights do not depend on the barrier ----
    {
        const int g = lane >> 2, t = lane & 3;
        const bool vlo = g < hr, vhi = g + 8 < hr;
        const uint4 zero = make_uint4(0, 0, 0, 0);
        auto down_of = [&](int i, int& len) -> const T* {  // row g, this lane's channels
            const bool shared = i < nsh;
            len = shared ? p.Is : p.I;
            const T* base = shared ? p.sdown : p.edown + (size_t)(ent_e[i] - p.expert_base) * H * p.I;
            return base + (size_t)(h0 + g) * len + 16 * t;
        };
        auto act_of = [&](int i) -> const T* {  // null: the column has no token
            const int pair = ent_pair[i * kWdCols + g];
            if (pair < 0) return nullptr;
            return (pair >= kWdPairs ? p.sact + (size_t)(pair - kWdPairs) * 3 * p.Is : p.act + (size_t)pair * 3 * p.I) + 16 * t;
        };
        uint4 wa[kWdDownAhead], wb[kWdDownAhead];
        uint4 fh[2], fm[2], fl[2];
        int len = 0, nlen = 0;
        const T* wrow = nullptr;
        int i = warp;
#pragma unroll
        for (int j = 0; j < kWdDownAhead; ++j) {
            wa[j] = zero;
            wb[j] = zero;
        }
        if (i < entries) {
            wrow = down_of(i, len);
            nlen = len;
#pragma unroll
            for (int j = 0; j < kWdDownAhead; j += 2) {
                if (vlo) ld_stream_2u4(wrow + 32 * j, wa[j], wa[j + 1]);
                if (vhi) ld_stream_2u4(wrow + 8 * len + 32 * j, wb[j], wb[j + 1]);
            }
        }
        if (!grid_barrier(p.ctl, ncta, 1u, kStatusMoeBarrier2, &s_flag)) return;
        if (tid == 0) barrier_finish(p.ctl, ncta);
        if (tracer) trace_stamp(p.ctl, 6);

        const T* arow = nullptr;
        auto fetch_act = [&](int slot, const T* a, int n) {  // 32 channels of an activation vector of length n
            fh[slot] = zero; fm[slot] = zero; fl[slot] = zero;
            if (a != nullptr) {
                fh[slot] = __ldcg(reinterpret_cast<const uint4*>(a));
                fm[slot] = __ldcg(reinterpret_cast<const uint4*>(a + n));
                fl[slot] = __ldcg(reinterpret_cast<const uint4*>(a + 2 * n));
            }
        };
        if (i < entries) {
            arow = act_of(i);
            fetch_act(0, arow, len);
            fetch_act(1, arow == nullptr ? arow : arow + 8, len);
        }
        bool odd = false;  // an element of this warp came out as NaN
#pragma unroll 1
        for (; i < entries; i += kWdWarps) {
            float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
            const int R = len / (32 * kWdDownAhead);  // whole rounds of slices
#pragma unroll 1
            for (int r = 0; r < R; ++r) {
                const bool same = r + 1 < R;
                const bool more = same || i + kWdWarps < entries;
                const T* nact = (arow != nullptr) ? arow + 32 * kWdDownAhead : nullptr;
                if (same) {
                    wrow += 32 * kWdDownAhead;
                } else if (more) {
                    wrow = down_of(i + kWdWarps, nlen);
                    nact = act_of(i + kWdWarps);
                }
                const T* whi = wrow + 8 * nlen;
#pragma unroll
                for (int j = 0; j < kWdDownAhead; j += 2) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_slice32<T>(s0, s1, wa[j + q], wb[j + q], fl[q]);
                        mma_slice32<T>(s0, s1, wa[j + q], wb[j + q], fm[q]);
                        mma_slice32<T>(s0, s1, wa[j + q], wb[j + q], fh[q]);
                        add_tile(d0, s0);
                        add_tile(d1, s1);
                        if (j + 2 < kWdDownAhead) fetch_act(q, arow == nullptr ? arow : arow + 32 * (j + 2) + 8 * q, len);
                        else if (more) fetch_act(q, nact == nullptr ? nact : nact + 8 * q, nlen);
                    }
                    if (more) {
                        if (vlo) ld_stream_2u4(wrow + 32 * j, wa[j], wa[j + 1]);
                        if (vhi) ld_stream_2u4(whi + 32 * j, wb[j], wb[j + 1]);
                    }
                }
                arow = nact;
            }
            // rows g and g + 8, columns 2t and 2t + 1
            add_tile(d0, d1);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int pair = ent_pair[i * kWdCols + 2 * t + c];
                if (pair >= 0) {
                    if (vlo) part_out[pair * p.hr_max + g] = d0[c];
                    if (vhi) part_out[pair * p.hr_max + g + 8] = d0[2 + c];
                    odd |= (vlo && isnan(d0[c])) || (vhi && isnan(d0[2 + c]));
                }
            }
            len = nlen;
        }
        if (__any_sync(kFullMask, odd)) wide_down_again(p, part_out, ent_e, ent_pair, entries, nsh, h0, hr, warp, lane);
    }
    if (tracer) trace_stamp(p.ctl, 7);
    __syncthreads();

    // ---- combine in slot order, residual, one rounding: item = (token, row) ----
    for (int item = tid; item < p.ntok * 16; item += kWdThreads) {
        const int b = item >> 4, j = item & 15;
        if (j < hr) {
            double vd = 0.0;
#pragma unroll 4
            for (int k = 0; k < p.K; ++k) {
                const int pair = b * kWdSlots + k;
                const int e = s_pair_e[pair];
                if (e >= p.expert_base && e < p.expert_base + p.local_experts) vd = fma((double)s_pair_w[pair], (double)part_out[pair * p.hr_max + j], vd);
            }
            if (p.Is > 0) vd += part_out[(kWdPairs + b) * p.hr_max + j];
            const float v = (float)vd;
            const size_t o = (size_t)b * H + h0 + j;
            if (p.partial_out) p.partial_out[o] = v;
            else p.out[o] = from_float<T>(p.add_residual ? v + to_float<T>(p.x[o]) : v);
        }
    }
    if (tracer) trace_stamp(p.ctl, 9);
}

// Launches the kernel, up to 32 tokens per launch, when the call suits it and sets *handled; otherwise leaves *handled false (no error).
int moe_decode_wide_launch(const mk36_moe_args* a, const mk36_comm* comm, void* workspace, size_t workspace_bytes, cudaStream_t stream,
                           bool* handled) {
    *handled = false;
    if (a->dtype != MK36_BF16) return MK36_OK;          // f16 terms cannot hold every fp32 activation
    if (comm && comm->world > 1) return MK36_OK;        // the exchange buffers are laid out for eight tokens
    const int H = a->hidden, E = a->experts, K = a->top_k, I = a->intermediate, Is = a->shared_intermediate;
    if (K <= 0 || K > kWdSlots || E <= 0 || E > 32 * kStTopkPerLane || I <= 0 || Is < 0) return MK36_OK;
    // slices in whole rounds
    if (H % (32 * kWdQuadWarps * kWdAhead) != 0 || H > 8 * 32 * kWdPieces || I % (32 * kWdDownAhead) != 0 || Is % (32 * kWdDownAhead) != 0)
        return MK36_OK;
    const void* ptrs[] = {a->x, a->norm_weight, a->router_weight, a->expert_gate, a->expert_up, a->expert_down,
                          a->shared_gate, a->shared_up, a->shared_down};
    for (const void* q : ptrs)
        if ((reinterpret_cast<uintptr_t>(q) & 31u) != 0) return MK36_OK;  // 32-byte loads
    const DeviceInfo* dev = current_device_info();
    if (!dev) return MK36_ERR_LAUNCH;
    const int ncta = dev->sm_count;
    const int hr_max = (H + ncta - 1) / ncta;
    if (hr_max > 16 || (E + ncta - 1) / ncta > kWdRouterRows) return MK36_OK;
    if ((long long)(kWdMaxEntries) * (I / 8) >= (1ll << 30) || (long long)kWdMaxTokens * (Is / 8) >= (1ll << 30)) return MK36_OK;
    const int launches = (a->batch + kWdMaxTokens - 1) / kWdMaxTokens;
    const int tb = (a->batch + launches - 1) / launches;  // the tokens shared out evenly

    MoeWideParams p;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        off = align_up(off, 128);
        const size_t at = off;
        off += bytes;
        return (int)at;
    };
    p.off_part = take((size_t)2 * kWdWarps * 32 * 16);
    p.off_row = take((size_t)kWdRouterRows * H * 2);
    p.off_norm = take((size_t)H * 2);
    p.off_slot = take((size_t)E * kWdMaxTokens);
    p.off_emask = take((size_t)E * 4);
    p.off_ent_e = take((size_t)kWdMaxEntries * 4);
    p.off_ent_m = take((size_t)kWdMaxEntries * 4);
    p.off_ent_tok = take((size_t)kWdMaxEntries * kWdCols);
    p.off_ent_pair = take((size_t)kWdMaxEntries * kWdCols * 2);
    p.off_pair_e = take((size_t)kWdPairs * 4);
    p.off_pair_w = take((size_t)kWdPairs * 4);
    const size_t x_bytes = (size_t)tb * (H + kWdPad) * 2, part_bytes = (size_t)(kWdPairs + kWdMaxTokens) * hr_max * 4;
    p.off_x = take(x_bytes > part_bytes ? x_bytes : part_bytes);
    const size_t smem = off;
    if (smem + 1024 > (size_t)dev->max_smem_optin) return MK36_OK;

    const size_t logit_bytes = align_up((size_t)kWdMaxTokens * E * 4, 256), act_bytes = align_up((size_t)kWdPairs * 3 * I * 2, 256);
    const size_t scratch = logit_bytes + act_bytes + align_up((size_t)kWdMaxTokens * 3 * (Is > 0 ? Is : 1) * 2, 256);
    // scratch ends below the mailboxes; a smaller workspace takes another kernel
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 || workspace_bytes < kControlBytes + scratch ||
        kControlBytes + scratch > kMailboxOffset)
        return MK36_OK;

    p.norm_w = static_cast<const __nv_bfloat16*>(a->norm_weight);
    p.router_w = static_cast<const __nv_bfloat16*>(a->router_weight);
    p.egate = static_cast<const __nv_bfloat16*>(a->expert_gate);
    p.eup = static_cast<const __nv_bfloat16*>(a->expert_up);
    p.edown = static_cast<const __nv_bfloat16*>(a->expert_down);
    p.sgate = static_cast<const __nv_bfloat16*>(a->shared_gate);
    p.sup = static_cast<const __nv_bfloat16*>(a->shared_up);
    p.sdown = static_cast<const __nv_bfloat16*>(a->shared_down);
    p.ctl = static_cast<Control*>(workspace);
    unsigned char* sc = static_cast<unsigned char*>(workspace) + kControlBytes;
    p.logits = reinterpret_cast<float*>(sc);
    p.act = reinterpret_cast<__nv_bfloat16*>(sc + logit_bytes);
    p.sact = reinterpret_cast<__nv_bfloat16*>(sc + logit_bytes + act_bytes);
    p.H = H; p.E = E; p.K = K; p.I = I; p.Is = Is;
    p.expert_base = a->expert_base;
    p.local_experts = a->local_experts;
    p.add_residual = a->add_residual;
    p.eps = a->eps;
    p.hr_max = hr_max;
    p.fd_tiles = make_fastdiv(I / 8);
    p.fd_stiles = make_fastdiv(Is > 0 ? Is / 8 : 1);

    const void* kernel = (const void*)moe_decode_wide_kernel;
    const int rc_smem = ensure_dynamic_smem(kernel, smem);
    if (rc_smem != MK36_OK) return rc_smem;
    for (int b0 = 0; b0 < a->batch; b0 += tb) {
        p.ntok = (a->batch - b0 < tb) ? (a->batch - b0) : tb;
        p.x = static_cast<const __nv_bfloat16*>(a->x) + (size_t)b0 * H;
        p.out = a->out ? static_cast<__nv_bfloat16*>(a->out) + (size_t)b0 * H : nullptr;
        p.partial_out = a->partial_out ? a->partial_out + (size_t)b0 * H : nullptr;
        p.indices = reinterpret_cast<long long*>(a->indices) + (size_t)b0 * K;
        p.route_w = a->route_weights + (size_t)b0 * K;
        void* params[] = {&p};
        const int rc = launch_cooperative(kernel, dim3(ncta), dim3(kWdThreads), smem, stream, params, "moe_decode(wide)");
        if (rc != MK36_OK) return rc;
    }
    *handled = true;
    return MK36_OK;
}

}  // namespace mk36
