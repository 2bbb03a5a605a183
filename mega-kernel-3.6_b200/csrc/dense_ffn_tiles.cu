// Dense SwiGLU FFN decode for two to eight tokens on sm_100a (2-byte dtypes): tensor-core tiles fed by a
// bulk-copy ring.
//
// out = x + Wd (silu(Wg n) * (Wu n)),  n = RMSNorm(x)       (mega_kernel_qwen36/reference.py:65-88)
//
// The weight stream bounds it (535 MB at hidden 5120, intermediate 17408).  dense_ffn_mma.cu loads the
// weights into fragments with register loads and stops at 4.0 TB/s: an SM cannot keep enough such loads
// outstanding.  Here the copy engine keeps four stages of 32 KB in flight per SM and the registers hold
// only what is being multiplied: eight tokens at that shape 133 -> 115 us (4.6 TB/s), bf16.
//
//   stage    up to 16 weight rows by up to 1024 columns, one bulk copy per row; rows lie 16 bytes apart
//            modulo 128, so that the fragment loads (eight rows, four 16-byte pieces) meet all banks
//   phase A  tile = up to eight gate rows and the matching up rows, the 16 rows of mma.sync.m16n8k16; the
//            tokens are its eight columns.  The eight consumer warps take every eighth 32-wide slice of a
//            stage, keep their accumulators over the tile's stages and meet in shared memory at its end;
//            silu(g) * u is stored as a high and a low half in the storage dtype
//   grid barrier (the producer warp is already streaming down rows)
//   phase C  the CTA's output rows in up to three tiles, all of them for one column range before the next,
//            so that a warp's activation fragments serve three stages
//   combine  in shared memory; residual, rounding, store (or the cross-GPU exchange)
//
// Sums: a stage's products are one chain of MMAs from zero, and the stages are added up in fp32.  As one chain over all
// stages, f16 at an eighth of the width was further from the 64-bit sum than the register-staged kernel (relative error
// 1.15e-6 against 0.97e-6); this way 4.1e-7, and bf16 at the whole width 2.5e-6 against 6.4e-6.  It costs 1 % (27B, four
// tokens 109.1 -> 110.5 us).
//
// Fragment conventions: mk36_mma.cuh.  Ring protocol: mk36_ring.cuh, every consumer warp observes and
// releases every stage.
#include "mk36_comm.cuh"
#include "mk36_mma.cuh"
#include "mk36_ring.cuh"

namespace mk36 {

constexpr int kDtWarps = 8;   // consumers; one more warp produces
constexpr int kDtConsumers = kDtWarps * 32;
constexpr int kDtThreads = kDtConsumers + 32;
constexpr int kDtMaxTokens = 8;
constexpr int kDtMaxStages = 6;
constexpr int kDtPad = 8;     // elements
constexpr int kDtStageBytes = 16 * (1024 + kDtPad) * 2;
constexpr int kDtMaxTiles = 3;     // 16-row output tiles per CTA
constexpr int kDtDownSlices = 5;   // 32-wide slices of a phase C stage per warp: their activation fragments stay in registers

struct DenseTilesParams {
    const void* x;
    const void* norm_w;
    const void* gate;
    const void* up;
    const void* down;
    void* out;
    float* partial_out;
    Control* ctl;
    void* act_hi;  // [8][I] in the storage dtype: silu(g) * u = hi + lo
    void* act_lo;
    float* act;    // [8][I]: silu(g) * u where hi is not finite (f16 ends at 65504), unwritten elsewhere
    int ntok, H, I, add_residual;
    float eps;
    int pa, kca;   // phase A: channels per tile, columns per stage
    int pc, kcc;   // phase C: rows per tile, columns per stage
    int nstages, off_red, off_x, off_ring;
    CommParams comm;
};

// Output row `row` of a token whose down product came out as an infinity or NaN, from the activations' values.
template <typename T>
static __device__ __noinline__ float dense_tiles_again(const DenseTilesParams& p, int token, int row) {
    const size_t I = (size_t)p.I;
    const T* hi = static_cast<const T*>(p.act_hi) + token * I;
    const T* lo = static_cast<const T*>(p.act_lo) + token * I;
    const float* whole = p.act + token * I;
    return down_element_again(static_cast<const T*>(p.down) + (size_t)row * I, p.I, [=](int k) {
        const float h = to_float<T>(__ldcg(hi + k));
        return fabsf(h) < INFINITY ? h + to_float<T>(__ldcg(lo + k)) : __ldcg(whole + k);
    });
}

template <typename T>
__global__ void __launch_bounds__(kDtThreads, 1) dense_ffn_tiles_kernel(const __grid_constant__ DenseTilesParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_flag;
    __shared__ int s_abort;
    __shared__ unsigned s_step;
    __shared__ float s_part[kDtWarps];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int cta = blockIdx.x, ncta = gridDim.x;
    const bool exchange = p.comm.world > 1;
    const bool tracer = (cta == 0 && tid == 0);

    unsigned long long* full_bar = reinterpret_cast<unsigned long long*>(smem);
    unsigned long long* empty_bar = full_bar + kDtMaxStages;
    T* xs = reinterpret_cast<T*>(smem + p.off_x);  // [8][H + pad], tokens beyond ntok are zero
    unsigned char* ring = smem + p.off_ring;
    const int R = p.nstages;
    const size_t H = (size_t)p.H, I = (size_t)p.I;
    const size_t xstride = H + kDtPad;

    const int c0 = (int)(((long long)p.I * cta) / ncta), c1 = (int)(((long long)p.I * (cta + 1)) / ncta);
    const int h0 = (int)(((long long)p.H * cta) / ncta), h1 = (int)(((long long)p.H * (cta + 1)) / ncta);
    const int hr = h1 - h0;
    const int ksteps_a = (p.H + p.kca - 1) / p.kca, ksteps_c = (p.I + p.kcc - 1) / p.kcc;
    const int tiles_c = (hr + p.pc - 1) / p.pc;

    if (tracer) trace_stamp(p.ctl, 0);
    if (tid < 2 * kDtMaxStages) mbar_init(&full_bar[tid], tid >= kDtMaxStages ? kDtWarps : 1);
    if (tid == 0) {
        s_abort = 0;
        s_step = exchange ? comm_read_step(p.comm) : 0u;
    }
    if (tid < 32) mbar_init_fence();
    __syncthreads();

    // =====================================================================================
    // Producer warp: one row per lane
    // =====================================================================================
    if (warp == kDtWarps) {
        // nothing is issued on a workspace whose status is set (a CTA that leaves must have no copy in flight)
        int dirty = 0;
        if (lane == 0) {
            dirty = ld_volatile_s32(&p.ctl->status);
            if (dirty != 0) *(volatile int*)&s_abort = 1;
        }
        if (__shfl_sync(kFullMask, dirty, 0) != 0) return;
        bool ok = true;
        int stage = 0, use = 0;
        // a stage of `rows` rows, `width` columns each; `src` is this lane's row (null: none), lane l fills row l
        auto issue = [&](const T* src, int rows, int width, int kc) {
            if (lane == 0) {
                if (use > 0) ok = mbar_wait(&empty_bar[stage], (unsigned)(use - 1) & 1u, &s_abort);
                if (ok) mbar_arrive_expect_tx(&full_bar[stage], (unsigned)(rows * width * (int)sizeof(T)));
            }
            ok = __shfl_sync(kFullMask, ok ? 1 : 0, 0) != 0;
            if (ok && src != nullptr)
                bulk_copy_g2s(ring + (size_t)stage * kDtStageBytes + (size_t)lane * (kc + kDtPad) * sizeof(T), src,
                              (unsigned)(width * (int)sizeof(T)), &full_bar[stage]);
            if (++stage == R) { stage = 0; ++use; }
        };
        for (int first = c0; first < c1 && ok; first += p.pa) {
            const int count = min(p.pa, c1 - first);
            const T* row = nullptr;  // lanes [0, count): gate rows, [pa, pa + count): up rows
            if (lane < count) row = static_cast<const T*>(p.gate) + (size_t)(first + lane) * H;
            else if (lane >= p.pa && lane < p.pa + count) row = static_cast<const T*>(p.up) + (size_t)(first + lane - p.pa) * H;
            for (int k = 0; k < ksteps_a && ok; ++k)
                issue(row == nullptr ? row : row + (size_t)k * p.kca, 2 * count, min(p.kca, p.H - k * p.kca), p.kca);
        }
        for (int k = 0; k < ksteps_c && ok; ++k) {
            for (int i = 0; i < tiles_c && ok; ++i) {
                const int first = h0 + i * p.pc, count = min(p.pc, h1 - first);
                const T* row = (lane < count) ? static_cast<const T*>(p.down) + (size_t)(first + lane) * I + (size_t)k * p.kcc : nullptr;
                issue(row, count, min(p.kcc, p.I - k * p.kcc), p.kcc);
            }
        }
        if (lane == 0) {
            if (!ok) {
                atomicCAS(&p.ctl->status, 0, kStatusMoeRingProducer);
                if (--stage < 0) { stage = R - 1; --use; }  // the stage that was not filled
            }
            ring_drain(full_bar, R, stage, use);
        }
        return;
    }

    // =====================================================================================
    // Consumer warps
    // =====================================================================================
    const T* x = static_cast<const T*>(p.x);
    const T* nw = static_cast<const T*>(p.norm_w);

    // ---- RMSNorm; the eight warps are shared out over the tokens (8, 4, 2 or 1 warps per token) ----
    {
        int tp2 = 1;
        while (tp2 < p.ntok) tp2 <<= 1;
        const int wpt = kDtWarps / tp2;  // warps per token
        const int b = warp / wpt, part = warp - b * wpt;
        const int nchunk = p.H >> 3, stride = wpt * 32;
        const bool live = b < p.ntok;
        const T* xr = x + (size_t)(live ? b : 0) * H;
        float ss = 0.0f;
        if (live) {
#pragma unroll 4
            for (int c = part * 32 + lane; c < nchunk; c += stride) {
                Chunk8<T> v;
                v.raw = *reinterpret_cast<const uint4*>(xr + 8 * c);
                float f[8];
                unpack8(v, f);
#pragma unroll
                for (int i = 0; i < 8; ++i) ss = fmaf(f[i], f[i], ss);
            }
        }
        ss = warp_sum(ss);
        if (lane == 0) s_part[warp] = ss;
        for (int idx = tid; idx < (kDtMaxTokens - p.ntok) * (int)(xstride >> 3); idx += kDtConsumers)
            *reinterpret_cast<uint4*>(xs + (size_t)p.ntok * xstride + 8 * (size_t)idx) = make_uint4(0, 0, 0, 0);
        named_barrier(1, kDtConsumers);
        if (live) {
            float tot = 0.0f;
            for (int w = 0; w < wpt; ++w) tot += s_part[b * wpt + w];
            const float rstd = 1.0f / sqrtf(tot / (float)p.H + p.eps);
            T* dst = xs + (size_t)b * xstride;
#pragma unroll 4
            for (int c = part * 32 + lane; c < nchunk; c += stride) {
                Chunk8<T> v, w;
                v.raw = *reinterpret_cast<const uint4*>(xr + 8 * c);
                w.raw = *reinterpret_cast<const uint4*>(nw + 8 * c);
                float f[8], wf[8];
                unpack8(v, f);
                unpack8(w, wf);
                T o[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = from_float<T>(__fmul_rn(__fmul_rn(f[i], rstd), wf[i]));
                *reinterpret_cast<uint4*>(dst + 8 * c) = *reinterpret_cast<const uint4*>(o);
            }
        }
        named_barrier(1, kDtConsumers);
    }
    if (tracer) trace_stamp(p.ctl, 1);

    bool ok = true;
    int stage = 0, use = 0;
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
        if (++stage == R) { stage = 0; ++use; }
    };

    // ---- phase A ----
    T* act_hi = static_cast<T*>(p.act_hi);
    T* act_lo = static_cast<T*>(p.act_lo);
    int buffer = 0;
#pragma unroll 1
    for (int first = c0; first < c1; first += p.pa) {
        const int count = min(p.pa, c1 - first);
        const int rl = min(g, count - 1);  // rows beyond the tile repeat its last one: not stored
        float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int k = 0; k < ksteps_a; ++k) {
            ok = mbar_wait(&full_bar[stage], (unsigned)use & 1u, &s_abort);
            if (!ok) break;
            const T* sbase = reinterpret_cast<const T*>(ring + (size_t)stage * kDtStageBytes);
            const T* alo = sbase + (size_t)rl * (p.kca + kDtPad) + 8 * t;
            const T* ahi = sbase + (size_t)(p.pa + rl) * (p.kca + kDtPad) + 8 * t;
            const T* bx = xs + (size_t)g * xstride + (size_t)k * p.kca + 8 * t;
            const int width = min(p.kca, p.H - k * p.kca);
            float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int c = 32 * warp; c < width; c += 32 * kDtWarps) mma_slice32<T>(s0, s1, lds128(alo + c), lds128(ahi + c), lds128(bx + c));
            release();
            add_tile(d0, s0);
            add_tile(d1, s1);
        }
        // The warps' shares of the tile meet; two buffers, so one barrier per tile.  A warp whose wait has run out comes to
        // every tile's barrier like the others: the barrier has no limit, and they may be some tiles from giving up.  What
        // such a CTA stores stays in the scratch buffer, because it does not arrive at the grid barrier.
        float* red = reinterpret_cast<float*>(smem + p.off_red) + buffer * (kDtWarps * 128);
        float* mine = red + warp * 128;
        *reinterpret_cast<float2*>(mine + g * 8 + 2 * t) = make_float2(d0[0] + d1[0], d0[1] + d1[1]);
        *reinterpret_cast<float2*>(mine + (g + 8) * 8 + 2 * t) = make_float2(d0[2] + d1[2], d0[3] + d1[3]);
        named_barrier(1, kDtConsumers);
        if (tid < 64) {
            const int tok = tid >> 3, ch = tid & 7;
            if (ch < count && tok < p.ntok) {
                float gv = 0.0f, uv = 0.0f;
#pragma unroll
                for (int w = 0; w < kDtWarps; ++w) {
                    gv += red[w * 128 + ch * 8 + tok];
                    uv += red[w * 128 + (ch + 8) * 8 + tok];
                }
                const float v = silu(gv) * uv;
                const T hi = from_float<T>(v);
                const bool fits = fabsf(to_float<T>(hi)) < INFINITY;
                const size_t at = (size_t)tok * I + first + ch;
                act_hi[at] = hi;
                act_lo[at] = from_float<T>(fits ? v - to_float<T>(hi) : 0.0f);
                if (!fits) p.act[at] = v;
            }
        }
        buffer ^= 1;
    }
    if (*(volatile int*)&s_abort != 0) atomicCAS(&p.ctl->status, 0, kStatusMoeRingConsumer);
    if (tracer) trace_stamp(p.ctl, 2);

    // ---- grid barrier: all activations are in the workspace ----
    named_barrier(1, kDtConsumers);
    if (tid == 0) {
        bool fine = (*(volatile int*)&s_abort == 0);  // set before the barrier by a warp whose wait has run out
        if (fine) {
            fine = barrier_wait(p.ctl, barrier_arrive(p.ctl, ncta, 0), kStatusDenseBarrier);
            if (fine) barrier_finish(p.ctl, ncta);
        }
        if (!fine) *(volatile int*)&s_abort = 1;
        s_flag = fine ? 1 : 0;
    }
    named_barrier(1, kDtConsumers);
    if (!s_flag) return;  // every consumer warp leaves; the producer sees the abort flag in its waits
    if (tracer) trace_stamp(p.ctl, 3);

    // ---- phase C: for each column range the CTA's row tiles in turn, against the same activation fragments ----
    float acc[kDtMaxTiles][2][4];
#pragma unroll
    for (int i = 0; i < kDtMaxTiles; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) { acc[i][j][0] = 0.f; acc[i][j][1] = 0.f; acc[i][j][2] = 0.f; acc[i][j][3] = 0.f; }
    {
        const bool col = g < p.ntok;  // columns beyond the batch are never stored
        const T* hrow = act_hi + (size_t)g * I + 8 * t;
        const T* lrow = act_lo + (size_t)g * I + 8 * t;
        uint4 bh[kDtDownSlices], bl[kDtDownSlices];
#pragma unroll
        for (int s = 0; s < kDtDownSlices; ++s) { bh[s] = make_uint4(0, 0, 0, 0); bl[s] = bh[s]; }
        auto fetch = [&](int s, int k) {  // this warp's slice s of column range k
            const int c = 32 * (warp + s * kDtWarps), at = k * p.kcc + c;
            if (col && c < p.kcc && at < p.I) {
                bh[s] = __ldcg(reinterpret_cast<const uint4*>(hrow + at));
                bl[s] = __ldcg(reinterpret_cast<const uint4*>(lrow + at));
            }
        };
#pragma unroll
        for (int s = 0; s < kDtDownSlices; ++s) fetch(s, 0);
#pragma unroll 1
        for (int k = 0; k < ksteps_c && ok; ++k) {
            const int width = min(p.kcc, p.I - k * p.kcc);
#pragma unroll
            for (int i = 0; i < kDtMaxTiles; ++i) {
                if (i < tiles_c && ok) {
                    ok = mbar_wait(&full_bar[stage], (unsigned)use & 1u, &s_abort);
                    if (ok) {
                        const int count = min(p.pc, hr - i * p.pc);
                        const T* sbase = reinterpret_cast<const T*>(ring + (size_t)stage * kDtStageBytes) + 8 * t;
                        const T* alo = sbase + (size_t)min(g, count - 1) * (p.kcc + kDtPad);
                        const T* ahi = sbase + (size_t)min(g + 8, count - 1) * (p.kcc + kDtPad);
                        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int s = 0; s < kDtDownSlices; ++s) {
                            const int c = 32 * (warp + s * kDtWarps);
                            if (c < width) {
                                const uint4 a = lds128(alo + c), b = lds128(ahi + c);
                                mma_slice32<T>(s0, s1, a, b, bl[s]);
                                mma_slice32<T>(s0, s1, a, b, bh[s]);
                            }
                        }
                        release();
                        add_tile(acc[i][0], s0);
                        add_tile(acc[i][1], s1);
                    }
                }
            }
            if (k + 1 < ksteps_c) {
#pragma unroll
                for (int s = 0; s < kDtDownSlices; ++s) fetch(s, k + 1);
            }
        }
    }
    if (!ok) atomicCAS(&p.ctl->status, 0, kStatusMoeRingConsumer);
    if (tracer) trace_stamp(p.ctl, 4);

    // ---- the warps' partial tiles meet over the token vectors, which are no longer needed ----
    float* red = reinterpret_cast<float*>(smem + p.off_x);
#pragma unroll
    for (int i = 0; i < kDtMaxTiles; ++i) {
        if (i < tiles_c) {
            float* mine = red + (warp * kDtMaxTiles + i) * 128;
            *reinterpret_cast<float2*>(mine + g * 8 + 2 * t) = make_float2(acc[i][0][0] + acc[i][1][0], acc[i][0][1] + acc[i][1][1]);
            *reinterpret_cast<float2*>(mine + (g + 8) * 8 + 2 * t) = make_float2(acc[i][0][2] + acc[i][1][2], acc[i][0][3] + acc[i][1][3]);
        }
    }
    named_barrier(1, kDtConsumers);
    if (*(volatile int*)&s_abort != 0 || !ok) return;
    T* out = static_cast<T*>(p.out);
    const unsigned step = s_step;
    for (int idx = tid; idx < hr * 8; idx += kDtConsumers) {
        const int r = idx >> 3, c = idx & 7;
        if (c >= p.ntok) continue;
        const int tile = r / p.pc, rr = r - tile * p.pc;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < kDtWarps; ++w) v += red[(w * kDtMaxTiles + tile) * 128 + rr * 8 + c];
        if (!(fabsf(v) < INFINITY)) v = dense_tiles_again<T>(p, c, h0 + r);
        const size_t o = (size_t)c * H + h0 + r;
        if (exchange) {
            comm_put(p.comm, step, o, v);
        } else if (p.partial_out) {
            p.partial_out[o] = v;
        } else {
            if (p.add_residual) v += to_float<T>(x[o]);
            out[o] = from_float<T>(v);
        }
    }
    if (exchange) {
        for (int idx = tid; idx < hr * 8; idx += kDtConsumers) {
            const int r = idx >> 3, c = idx & 7;
            if (c >= p.ntok) continue;
            const size_t o = (size_t)c * H + h0 + r;
            float v;
            if (!comm_get_sum(p.comm, p.ctl, step, o, &v)) continue;
            if (p.add_residual) v += to_float<T>(x[o]);
            out[o] = from_float<T>(v);
        }
        if (cta == 0 && tid == 0) comm_write_step(p.comm, step + 1u);  // every CTA read it before the grid barrier
    }
    if (tracer) trace_stamp(p.ctl, 5);
}

// Launches the kernel, eight tokens per launch, when the call suits it (2-byte dtype, aligned shapes, at least three
// stages beside the tokens) and sets *handled; otherwise leaves *handled false (no error).
int dense_ffn_tiles_launch(const mk36_dense_ffn_args* a, const mk36_comm* comm, void* workspace, size_t workspace_bytes, cudaStream_t stream,
                           bool* handled) {
    *handled = false;
    if (a->dtype != MK36_BF16 && a->dtype != MK36_F16) return MK36_OK;
    const int H = a->hidden, I = a->intermediate;
    if (H % 32 != 0 || I % 32 != 0) return MK36_OK;
    const void* ptrs[] = {a->x, a->norm_weight, a->gate_weight, a->up_weight, a->down_weight};
    for (const void* q : ptrs)
        if ((reinterpret_cast<uintptr_t>(q) & 15u) != 0) return MK36_OK;
    const DeviceInfo* dev = current_device_info();
    if (!dev) return MK36_ERR_LAUNCH;
    const int ncta = dev->sm_count;
    if (H < ncta || I < ncta) return MK36_OK;  // every CTA has a tile in both phases
    const int hr_max = (H + ncta - 1) / ncta, ch_max = (I + ncta - 1) / ncta;
    if (hr_max > 16 * kDtMaxTiles) return MK36_OK;

    DenseTilesParams p;
    size_t off = align_up(2 * kDtMaxStages * 8, 128);
    p.off_red = (int)off;
    off += 2 * kDtWarps * 128 * 4;
    p.off_x = (int)off;
    const size_t xs_bytes = (size_t)kDtMaxTokens * (H + kDtPad) * 2, red_bytes = (size_t)kDtWarps * kDtMaxTiles * 128 * 4;
    off = align_up(off + (xs_bytes > red_bytes ? xs_bytes : red_bytes), 128);
    p.off_ring = (int)off;
    int nstages = (int)(((long long)dev->max_smem_optin - (long long)off - 1024) / kDtStageBytes);
    if (nstages > kDtMaxStages) nstages = kDtMaxStages;
    if (nstages < 3) return MK36_OK;  // too little in flight to be worth it
    p.nstages = nstages;
    const size_t smem = off + (size_t)nstages * kDtStageBytes;
    // equal tiles, and as many columns per stage as fit beside the tile's rows
    const int tiles_a = (ch_max + 7) / 8, tiles_c = (hr_max + 15) / 16;
    p.pa = (ch_max + tiles_a - 1) / tiles_a;
    p.pc = (hr_max + tiles_c - 1) / tiles_c;
    p.kca = (kDtStageBytes / 2 / (2 * p.pa) - kDtPad) / 256 * 256;
    p.kcc = (kDtStageBytes / 2 / p.pc - kDtPad) / 256 * 256;
    if (p.kca > 4096) p.kca = 4096;
    if (p.kcc > 32 * kDtWarps * kDtDownSlices) p.kcc = 32 * kDtWarps * kDtDownSlices;

    int rc = comm_params_from(comm, H, &p.comm, "dense_ffn_decode");
    if (rc != MK36_OK) return rc;
    if (p.comm.world > 1 && (!a->out || a->partial_out))
        MK36_FAIL(MK36_ERR_INVALID_ARG, "dense_ffn_decode: the multi-GPU entry point writes `out` and takes no partial_out");
    // a smaller workspace takes the register-staged kernel, which needs half of it; scratch ends below the mailboxes
    const size_t act_bytes = align_up((size_t)kDtMaxTokens * I * 2, 256);
    if (!workspace || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 || workspace_bytes < kControlBytes + 4 * act_bytes ||
        kControlBytes + 4 * act_bytes > kMailboxOffset)
        return MK36_OK;

    p.norm_w = a->norm_weight;
    p.gate = a->gate_weight;
    p.up = a->up_weight;
    p.down = a->down_weight;
    p.ctl = static_cast<Control*>(workspace);
    p.act_hi = static_cast<unsigned char*>(workspace) + kControlBytes;
    p.act_lo = static_cast<unsigned char*>(workspace) + kControlBytes + act_bytes;
    p.act = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + kControlBytes + 2 * act_bytes);
    p.H = H;
    p.I = I;
    p.add_residual = a->add_residual;
    p.eps = a->eps;
    const void* kernel = (a->dtype == MK36_BF16) ? (const void*)dense_ffn_tiles_kernel<__nv_bfloat16> : (const void*)dense_ffn_tiles_kernel<__half>;
    rc = ensure_dynamic_smem(kernel, smem);
    if (rc != MK36_OK) return rc;
    for (int b0 = 0; b0 < a->batch; b0 += kDtMaxTokens) {
        p.ntok = (a->batch - b0 < kDtMaxTokens) ? (a->batch - b0) : kDtMaxTokens;
        p.x = static_cast<const unsigned char*>(a->x) + (size_t)b0 * H * 2;
        p.out = a->out ? static_cast<unsigned char*>(a->out) + (size_t)b0 * H * 2 : nullptr;
        p.partial_out = a->partial_out ? a->partial_out + (size_t)b0 * H : nullptr;
        void* params[] = {&p};
        rc = launch_cooperative(kernel, dim3(ncta), dim3(kDtThreads), smem, stream, params, "dense_ffn_decode(tiles)");
        if (rc != MK36_OK) return rc;
    }
    *handled = true;
    return MK36_OK;
}

}  // namespace mk36
