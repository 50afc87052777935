// Standalone quantize, in-place dequantize and low-rank factorisation kernels (sm_100a).
//
// Quantize: persistent CTAs, a head's 128 x 128 fp32 tile in the registers of one CTA, the next head's on its way into shared
// memory.  Dequantize: persistent CTAs that walk the heads, each head's checkpoint staged in shared memory.  Low-rank: one CTA
// of 256 threads per matrix, which stays in shared memory.
// Either way the in-place rewrite of a slot (fp32 state <-> packed 8-bit checkpoint) never reads what it has already
// overwritten.
#include "lq_linalg.cuh"

namespace lq {

// ------------------------------------------------------------------------------------------------------------------
// quantize
// ------------------------------------------------------------------------------------------------------------------
// One head = one 128 x 128 fp32 tile, held in REGISTERS by the 256 threads of a CTA (64 values each) from the moment it has
// arrived until its codes are stored; persistent CTAs, two per SM.  The tile is read from shared memory once, so that the
// buffer is free for the next head's 64 KB -- one bulk asynchronous copy, in flight during the whole of this head's
// arithmetic -- and every product of the subspace iteration works on registers with packed f32x2 multiply-adds (two fp32
// products per instruction, each rounded as the scalar one would be).
// Thread (warp w, lane): lc = lane % 16, lr = lane / 16 owns rows 16 w + 8 lr + i (i < 8) and columns 4 lc .. + 3, 64 + 4 lc .. + 3.
//   P = S^T Q: 8 rows are summed in the thread, two half-warps by one exchange, eight warps through shared memory.
//   Q = S P:   8 columns in the thread, sixteen lanes by halving exchanges; a warp ends with its own 16 rows.
// What bounds it: issue slots of the sixteen resident warps (R = 4: 14 400 warp instructions per head, a third of them the
// multiply-adds, issued in 39 % of the cycles); the previous form read the tile from shared memory for every product (32 000
// instructions per head, three CTAs per SM).  Dequantize + quantize of 8 192 GDN heads: 496 -> 390 us, of 416 heads 39 -> 36 us,
// of 1 536 KDA heads (R = 8, three iterations) 277 -> 214 us.
constexpr int QZ_TILE = 128 * 128 * 4;
template <int R>
__host__ __device__ constexpr int qz_smem_bytes() { return QZ_TILE + 8 * R * 128 * 4 + R * 128 * 4 + R * 128 * 8 + R * 128 * 4; }

struct QzTile {
    float2 s[8][4];                       // [row i][column pair]: pairs 0, 1 = columns 4 lc .. + 3; 2, 3 = 64 + 4 lc .. + 3
};
// partial products over the warp's 16 rows: part[w][r][c] = sum_row S[row][c] Q[row][r]; Qd: [128][R] values duplicated to pairs
template <int R>
__device__ __forceinline__ void qz_coldot(const QzTile& t, const float2* __restrict__ Qd, float* __restrict__ part, int warp, int lane) {
    const int lc = lane & 15, lr = lane >> 4;
    const float2* qrow = Qd + (16 * warp + 8 * lr) * R;
    float* out = part + warp * (R * 128) + 64 * lr + 4 * lc;
#pragma unroll 1
    for (int rb = 0; rb < R; rb += 4) {
        float2 acc[4][4];                 // [column pair][r]
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 qa = *reinterpret_cast<const float4*>(qrow + i * R + rb), qb = *reinterpret_cast<const float4*>(qrow + i * R + rb + 2);
            const float2 q[4] = {make_float2(qa.x, qa.y), make_float2(qa.z, qa.w), make_float2(qb.x, qb.y), make_float2(qb.z, qb.w)};
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[p][r] = i == 0 ? __fmul2_rn(t.s[i][p], q[r]) : __ffma2_rn(t.s[i][p], q[r], acc[p][r]);
        }
        // the half-warp lr keeps the columns 64 lr + 4 lc .. + 3
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 lo = acc[k >> 1][r], hi = acc[2 + (k >> 1)][r];
                const float a = (k & 1) ? lo.y : lo.x, b = (k & 1) ? hi.y : hi.x;
                v[k] = (lr ? b : a) + __shfl_xor_sync(0xffffffffu, lr ? a : b, 16);
            }
            *reinterpret_cast<float4*>(out + (rb + r) * 128) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}
// X[r][c] = sum over the eight warps' partials (all 256 threads), on request rounded to f16 values
template <int R>
__device__ __forceinline__ void qz_sum_parts(const float* __restrict__ part, float* __restrict__ X, int tid, bool round16) {
    constexpr int PT = R * 128 / NT_LA;   // outputs per thread: 2 or 4
    float a[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) a[k] = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if constexpr (PT == 2) {
            const float2 v = *reinterpret_cast<const float2*>(part + w * (R * 128) + 2 * tid);
            a[0] += v.x; a[1] += v.y;
        } else {
            const float4 v = *reinterpret_cast<const float4*>(part + w * (R * 128) + 4 * tid);
            a[0] += v.x; a[1] += v.y; a[2] += v.z; a[3] += v.w;
        }
    }
#pragma unroll
    for (int k = 0; k < PT; ++k) X[PT * tid + k] = round16 ? round_f16(a[k]) : a[k];
}
// X[r][row] = sum_c S[row][c] P[r][c]
template <int R>
__device__ __forceinline__ void qz_rowdot(const QzTile& t, const float* __restrict__ P, float* __restrict__ X, int warp, int lane) {
    const int lc = lane & 15, lr = lane >> 4;
    const bool b3 = lc & 8, b2 = lc & 4, b1 = lc & 2, b0 = lc & 1;
#pragma unroll 1
    for (int rb = 0; rb < R; rb += 4) {
        float v[4][4];                    // [row i or i + 4, by bit 3 of lc][r]
        float2 pv[4][4];                  // [r][column pair]
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 lo = *reinterpret_cast<const float4*>(P + (rb + r) * 128 + 4 * lc), hi = *reinterpret_cast<const float4*>(P + (rb + r) * 128 + 64 + 4 * lc);
            pv[r][0] = make_float2(lo.x, lo.y); pv[r][1] = make_float2(lo.z, lo.w);
            pv[r][2] = make_float2(hi.x, hi.y); pv[r][3] = make_float2(hi.z, hi.w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float2 x = __fmul2_rn(t.s[i][0], pv[r][0]), y = __fmul2_rn(t.s[i + 4][0], pv[r][0]);
#pragma unroll
                for (int p = 1; p < 4; ++p) {
                    x = __ffma2_rn(t.s[i][p], pv[r][p], x);
                    y = __ffma2_rn(t.s[i + 4][p], pv[r][p], y);
                }
                const float xs = x.x + x.y, ys = y.x + y.y;
                v[i][r] = (b3 ? ys : xs) + __shfl_xor_sync(0xffffffffu, b3 ? xs : ys, 8);
            }
        }
        float u[2][4], z[4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int r = 0; r < 4; ++r) u[i][r] = (b2 ? v[i + 2][r] : v[i][r]) + __shfl_xor_sync(0xffffffffu, b2 ? v[i][r] : v[i + 2][r], 4);
#pragma unroll
        for (int r = 0; r < 4; ++r) z[r] = (b1 ? u[1][r] : u[0][r]) + __shfl_xor_sync(0xffffffffu, b1 ? u[0][r] : u[1][r], 2);
        const float w0 = (b0 ? z[2] : z[0]) + __shfl_xor_sync(0xffffffffu, b0 ? z[0] : z[2], 1);
        const float w1 = (b0 ? z[3] : z[1]) + __shfl_xor_sync(0xffffffffu, b0 ? z[1] : z[3], 1);
        const int row = 16 * warp + 8 * lr + (b3 ? 4 : 0) + (b2 ? 2 : 0) + (b1 ? 1 : 0), r0 = rb + (b0 ? 2 : 0);
        X[r0 * 128 + row] = w0;
        X[(r0 + 1) * 128 + row] = w1;
    }
}
// Modified Gram-Schmidt of the R columns of X [R][128], warps 0 .. R - 1: warp j owns column j (lane = rows lane + 32 i) and takes
// the earlier columns out of it in the order 0, 1, ....  A round makes TWO columns a, b final: the five sums |a|^2, a.b, |b|^2, a.x,
// b.x (x: the warp's own column) come out of one reduction, and the products with b' = b - (q_a.b) q_a follow from them,
//   |b'|^2 = |b|^2 - (q_a.b)^2,  b'.x' = b.x - (q_a.b) (q_a.x),
// as long as b' keeps a quarter of |b|^2 -- then the differences cost two bits at most; where it does not, or where a sum left the
// range of fp32, they are summed from the vectors themselves, the pairwise form.  R / 2 rounds, R products side by side, in
// place of R (R + 1) / 2 reductions one after the other by one warp.  X is overwritten; on return x holds warp j's column.
template <int R>
__device__ __forceinline__ void qz_mgs(float* X, float (&x)[4], int warp, int lane) {
    if (warp >= R) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = X[warp * 128 + lane + 32 * i];
#pragma unroll 1
    for (int c = 0; c < R; c += 2) {
        float a[4], b[4], g[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = X[c * 128 + lane + 32 * i];
            b[i] = X[(c + 1) * 128 + lane + 32 * i];
            g[0] = fmaf(a[i], a[i], g[0]); g[1] = fmaf(a[i], b[i], g[1]); g[2] = fmaf(b[i], b[i], g[2]);
            g[3] = fmaf(a[i], x[i], g[3]); g[4] = fmaf(b[i], x[i], g[4]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 5; ++k) g[k] += __shfl_xor_sync(0xffffffffu, g[k], o);
        const bool in_range = fabsf(g[0]) + fabsf(g[1]) + fabsf(g[2]) + fabsf(g[3]) + fabsf(g[4]) <= 3.4e38f;
        const float na = rsqrtf(fmaxf(g[0], 1e-30f));
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] *= na;
        float t = g[1] * na, s = g[3] * na;
        if (!in_range) {                          // (the same in every lane) with the normalised column
            t = s = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) { t = fmaf(a[i], b[i], t); s = fmaf(a[i], x[i], s); }
            t = warp_sum(t);
            s = warp_sum(s);
        }
        float gb = fmaf(-t, t, g[2]), e = fmaf(-t, s, g[4]);
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = fmaf(-t, a[i], b[i]);
        if (warp > c)
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = fmaf(-s, a[i], x[i]);
        if (!in_range || !(gb >= 0.25f * g[2])) {
            gb = e = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) { gb = fmaf(b[i], b[i], gb); e = fmaf(b[i], x[i], e); }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { gb += __shfl_xor_sync(0xffffffffu, gb, o); e += __shfl_xor_sync(0xffffffffu, e, o); }
        }
        const float nb = rsqrtf(fmaxf(gb, 1e-30f));
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] *= nb;
        if (warp == c) {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = a[i];
        } else if (warp == c + 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = b[i];
        } else {
            e *= nb;
            if (!(fabsf(e) <= 3.4e38f)) {
                e = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) e = fmaf(b[i], x[i], e);
                e = warp_sum(e);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = fmaf(-e, b[i], x[i]);
            if (warp < c + 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) X[warp * 128 + lane + 32 * i] = x[i];
            }
        }
        if (warp < c + 2) return;                 // this warp's column is final
        named_bar(1 + (c >> 1), 32 * (R - c - 2));
    }
}

template <int R>
__global__ void __launch_bounds__(NT_LA, 2)
quantize_kernel(lq_dims d, char* __restrict__ ssm, float* __restrict__ Wbuf, float* __restrict__ Pbuf,
                uint16_t* __restrict__ Gbuf, int32_t* __restrict__ hcnt, const float* __restrict__ Q0,
                const int32_t* __restrict__ idx, int nheads, int kda, int iters) {
    extern __shared__ __align__(128) char qz_smem[];
    float* tile = reinterpret_cast<float*>(qz_smem);                   // [128][128] the head to come
    float* part = tile + 128 * 128;                                    // [8][R][128] partial products; also X = S P, |E| sums
    float* X = part + 8 * R * 128;                                     // [R][128] P^T, later U^T
    float2* Qd = reinterpret_cast<float2*>(X + R * 128);               // [128][R] Q, every value twice
    float* Q0s = reinterpret_cast<float*>(Qd + 128 * R);               // [128][R] the start of the iteration
    float* rsk = part + 8 * 128;                                       // [128] 1 / Sk (behind the sums of |E|, which part holds then)
    float* rowf = rsk + 128;                                           // [128] 127 / Sv
    __shared__ __align__(8) uint64_t load_bar;
    __shared__ int s_slot[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lc = lane & 15, lr = lane >> 4;
    const int first = blockIdx.x, stride = gridDim.x;

    auto slot_of = [&](int k) { const int p = first + k * stride; return p < nheads ? idx[p / d.HV] : 0; };
    auto usable = [&](int slot) { return slot > 0 && slot < d.NS; };
    auto fetch = [&](int k, int slot) {   // (thread 0)
        mbar_arrive_expect_tx(&load_bar, uint32_t(QZ_TILE));
        const char* src = head_base(ssm, d.SS, slot, (first + k * stride) % d.HV);
        bulk_g2s(qz_smem, src, QZ_TILE, &load_bar);
    };
    if (tid == 0) {
        mbar_init(&load_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        const int s0 = slot_of(0);
        s_slot[0] = s0;
        if (usable(s0)) fetch(0, s0);
    }
    for (int i = tid; i < R * 128; i += NT_LA) Q0s[i] = Q0[i];
    uint32_t phase = 0;
    for (int k = 0; first + k * stride < nheads; ++k) {
        __syncthreads();                  // the slot of this head is known; everything of the head before is done
        const int slot = s_slot[k & 1];
        const bool on = usable(slot);
        bool ok = true;
        QzTile t;
        if (on) {
#pragma unroll
            for (int u = 0; u < R / 2; ++u) {                          // Q <- Q0
                const float q = Q0s[tid + u * NT_LA];
                Qd[tid + u * NT_LA] = make_float2(q, q);
            }
            ok = warp_wait_bounded(&load_bar, phase);
            phase ^= 1u;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float* row = tile + (16 * warp + 8 * lr + i) * 128 + 4 * lc;
                const float4 lo = *reinterpret_cast<const float4*>(row), hi = *reinterpret_cast<const float4*>(row + 64);
                t.s[i][0] = make_float2(lo.x, lo.y); t.s[i][1] = make_float2(lo.z, lo.w);
                t.s[i][2] = make_float2(hi.x, hi.y); t.s[i][3] = make_float2(hi.z, hi.w);
            }
        }
        if (!__syncthreads_and(ok)) {     // the tile never came: nothing is written, the status word says why
            if (tid == 0) atomicOr(&g_status, ST_FLUSH_TIMEOUT);
            return;
        }
        // The tile is in registers and the next head's may come.  (It is only ever read through the generic proxy, and those reads
        // are behind the barrier: no proxy fence, which would also wait for the thread's stores to the head before.)
        auto fetch_next = [&] {           // (one thread)
            const int nx = slot_of(k + 1);
            s_slot[(k + 1) & 1] = nx;
            if (usable(nx)) fetch(k + 1, nx);
        };
        if (!on) {
            if (tid == 0) fetch_next();
            continue;
        }
        const int hv = (first + k * stride) % d.HV;
        char* base = head_base(ssm, d.SS, slot, hv);
        const int64_t sh = int64_t(slot) * d.HV + hv;

        // Work that does not wait for the arithmetic, done by four warps that have nothing to do in the first Gram-Schmidt (R = 4:
        // the warps without a column; R = 8: those whose columns are final first): the next head's copy, the window reset.
        auto aside = [&] {
            const int at = R == 4 ? tid - 128 : tid;
            if (at < 0 || at >= 128) return;
            if (at == 0) fetch_next();
            for (int j = at; j < d.L; j += 128) Wbuf[sh * d.L + j] = 0.f;
            if (kda) {
                Pbuf[sh * KD + at] = 0.f;
                uint4* g4 = reinterpret_cast<uint4*>(Gbuf + sh * d.L * KD);
                for (int i = at; i < d.L * KD / 8; i += 128) g4[i] = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);     // fp16 1.0
            } else if (at == 1) {
                Pbuf[sh] = 1.f;
            }
            if (at == 1) hcnt[sh] = 0;
        };
        // half steps: P = S^T Q, orthonormalised; Q = S P, orthonormalised; ...; U = S^T Q (one copy of each piece of code: a head
        // runs through this loop body once from a cold instruction cache)
#pragma unroll 1
        for (int hs = 0;; ++hs) {
            const bool to_q = hs & 1, last = hs >= 2 * iters;
            if (to_q) {
                qz_rowdot<R>(t, X, part, warp, lane);
            } else {
                qz_coldot<R>(t, Qd, part, warp, lane);
                __syncthreads();
                qz_sum_parts<R>(part, X, tid, last);
                if (last) {
                    if (hs == 0) aside();
                    break;
                }
            }
            __syncthreads();
            float x[4];
            qz_mgs<R>(to_q ? part : X, x, warp, lane);
            if (hs == 0) aside();
            if (!to_q) __syncthreads();   // (the raw columns are read until the last round is over)
            if (warp < R) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (to_q) Qd[(lane + 32 * i) * R + warp] = make_float2(x[i], x[i]);
                    else X[warp * 128 + lane + 32 * i] = x[i];
                }
            }
            __syncthreads();
        }
        __syncthreads();

        // residual E = S - Q U^T in place (one factor at a time, fused multiply-add), column sums of |E|
#pragma unroll 1
        for (int rb = 0; rb < R; rb += 4) {
            float2 u[4][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 lo = *reinterpret_cast<const float4*>(X + (rb + r) * 128 + 4 * lc), hi = *reinterpret_cast<const float4*>(X + (rb + r) * 128 + 64 + 4 * lc);
                u[r][0] = make_float2(lo.x, lo.y); u[r][1] = make_float2(lo.z, lo.w);
                u[r][2] = make_float2(hi.x, hi.y); u[r][3] = make_float2(hi.z, hi.w);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2* qrow = Qd + (16 * warp + 8 * lr + i) * R + rb;
                const float4 qa = *reinterpret_cast<const float4*>(qrow), qb = *reinterpret_cast<const float4*>(qrow + 2);
                // (both factors as they are stored: U was rounded to f16 as it was summed)
                const float qv[4] = {-round_f16(qa.x), -round_f16(qa.z), -round_f16(qb.x), -round_f16(qb.z)};
                const float2 q[4] = {make_float2(qv[0], qv[0]), make_float2(qv[1], qv[1]), make_float2(qv[2], qv[2]), make_float2(qv[3], qv[3])};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int p = 0; p < 4; ++p) t.s[i][p] = __ffma2_rn(q[r], u[r][p], t.s[i][p]);
            }
        }
        {
            float cs[8];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                cs[2 * p] = fabsf(t.s[0][p].x); cs[2 * p + 1] = fabsf(t.s[0][p].y);
#pragma unroll
                for (int i = 1; i < 8; ++i) { cs[2 * p] += fabsf(t.s[i][p].x); cs[2 * p + 1] += fabsf(t.s[i][p].y); }
            }
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = (lr ? cs[4 + j] : cs[j]) + __shfl_xor_sync(0xffffffffu, lr ? cs[j] : cs[4 + j], 16);
            *reinterpret_cast<float4*>(part + warp * 128 + 64 * lr + 4 * lc) = make_float4(v[0], v[1], v[2], v[3]);
        }
        __syncthreads();
        if (tid < 128) {
            float cs = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) cs += part[w * 128 + tid];
            const float skv = fmaxf(sqrtf(cs / float(VD)), EPS);
            rsk[tid] = 1.0f / skv;
            reinterpret_cast<float*>(base + CK_SK)[tid] = skv;
        }
        {                                 // the factors, two values per word: a row is 64 words of U^T and 64 of Q^T
            uint32_t* uq = reinterpret_cast<uint32_t*>(base + CK_UQ);
#pragma unroll
            for (int u = 0; u < R / 4; ++u) {
                const int r = (tid >> 6) + 4 * u, e = tid & 63;
                const __half2 hu = __floats2half2_rn(X[r * 128 + 2 * e], X[r * 128 + 2 * e + 1]);
                const __half2 hq = __floats2half2_rn(Qd[2 * e * R + r].x, Qd[(2 * e + 1) * R + r].x);
                uq[r * 128 + e] = *reinterpret_cast<const uint32_t*>(&hu);
                uq[r * 128 + 64 + e] = *reinterpret_cast<const uint32_t*>(&hq);
            }
        }
        __syncthreads();

        // Row scales and codes: Sv[v] = max(max_c |E| (1 / Sk), EPS), code = rint(E (1 / Sk) (127 / Sv)), which is the reference's
        // rint(E / (Sk Sv) * 127) (leapquant/kernels.py:2218-2229) wherever that lies further than 1e-4 code units from a rounding
        // boundary: either form carries at most four fp32 roundings of a value of at most 127.  |E (1 / Sk)| <= Sv, so the clamp
        // to +-127 never acts.  The sum with 1.5 * 2^23 rounds, and its low mantissa byte is the code in two's complement.
        float rm[8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float2 k2 = *reinterpret_cast<const float2*>(rsk + (p >> 1) * 64 + 4 * lc + 2 * (p & 1));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                t.s[i][p] = __fmul2_rn(t.s[i][p], k2);
                const float m = fmaxf(fabsf(t.s[i][p].x), fabsf(t.s[i][p].y));
                rm[i] = p == 0 ? m : fmaxf(rm[i], m);
            }
        }
        // the row maximum over sixteen lanes: lane bits 3..1 pick the row, bit 0 is folded last
        const bool b3 = lc & 8, b2 = lc & 4, b1 = lc & 2;
#pragma unroll
        for (int i = 0; i < 4; ++i) rm[i] = fmaxf(b3 ? rm[i + 4] : rm[i], __shfl_xor_sync(0xffffffffu, b3 ? rm[i] : rm[i + 4], 8));
#pragma unroll
        for (int i = 0; i < 2; ++i) rm[i] = fmaxf(b2 ? rm[i + 2] : rm[i], __shfl_xor_sync(0xffffffffu, b2 ? rm[i] : rm[i + 2], 4));
        rm[0] = fmaxf(b1 ? rm[1] : rm[0], __shfl_xor_sync(0xffffffffu, b1 ? rm[0] : rm[1], 2));
        rm[0] = fmaxf(rm[0], __shfl_xor_sync(0xffffffffu, rm[0], 1));
        {
            const int row = 16 * warp + 8 * lr + (lc >> 1);
            const float svv = fmaxf(rm[0], EPS);
            if (!(lc & 1)) {
                reinterpret_cast<float*>(base + CK_SV)[row] = svv;
                rowf[row] = QMAX / svv;
            }
        }
        __syncwarp();
        uint32_t* codes = reinterpret_cast<uint32_t*>(base + CK_CODES) + (16 * warp + 8 * lr) * 32 + lc;
        const float2 mg = make_float2(RNE_MAGIC, RNE_MAGIC);
        const float* rf = rowf + 16 * warp + 8 * lr;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float rv = rf[i];
            const float2 rv2 = make_float2(rv, rv);
            float2 z[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) z[p] = __ffma2_rn(t.s[i][p], rv2, mg);
            codes[i * 32] = pack4(__float_as_uint(z[0].x), __float_as_uint(z[0].y), __float_as_uint(z[1].x), __float_as_uint(z[1].y));
            codes[i * 32 + 16] = pack4(__float_as_uint(z[2].x), __float_as_uint(z[2].y), __float_as_uint(z[3].x), __float_as_uint(z[3].y));
        }

    }
}

// four 8 x 8 b16 tiles, transposed: lane l supplies the address of row l % 8 of tile l / 8 and receives, of each tile, the
// elements (2 (l % 4), l / 4) and (2 (l % 4) + 1, l / 4)
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}

// ------------------------------------------------------------------------------------------------------------------
// dequantize in place
// ------------------------------------------------------------------------------------------------------------------
// S[v][c] = (q8 / 127 Sk[c] Sv[v] + sum_r Q_r[v] U_r[c]) p pc[c] + sum_{j<h} (w_j u_j[v]) (k_j[c] D_j[c])   (leapquant/kernels.py:2105-2117;
// KDA: leapquant/state.py:118-128).  The constants are folded into the vectors first: skq[c] = Sk[c] / 127 (* pc[c]),
// svp[v] = Sv[v] p, Qp_r[v] = Q_r[v] p, Uc_r[c] = U_r[c] (* pc[c]).  The rank-R term runs on the tensor cores: Qp and Uc are
// split into a bf16 head and a bf16 remainder and the three products head x head, remainder x head, head x remainder are laid
// side by side along K of one `mma.sync.m16n8k16` (R = 4: K = 12 of 16; R = 8: two instructions), which keeps 16 bits of each
// factor -- 1e-5 of the term -- and replaces 4 R multiply-adds per element by an eighth of an instruction.  What is left per
// element is one conversion, one multiply, one fused multiply-add and h multiply-adds for the live window entries.  The
// values differ from the reference's evaluation order by a few units in the last place of fp32.
// Warp w owns rows 16 w .. 16 w + 15; lane (gid, tig) owns rows 16 w + gid, + 8 and, in each group of 16 columns, the four
// columns 4 tig .. 4 tig + 3: the two n-tiles of a group are mapped onto the columns so that every lane ends up with four
// contiguous ones (n index g of the first tile is column 4 (g / 2) + g % 2, of the second the same + 2).
// The window rows stay bf16 in shared memory (KDA keys: decayed, fp32).
// The kernel is persistent: two CTAs per SM, each taking the heads blockIdx.x, + gridDim.x, ...  A ninth warp runs ahead of
// the eight that compute: it looks up the slot, the window count and the scale of the heads to come (thirty-two at a time,
// one per lane) and brings each head's checkpoint -- codes, scales, factors: one contiguous piece -- into one of two stages
// with a bulk asynchronous copy, so that the three dependent trips to memory of a head (index -> counters -> checkpoint) are
// spent while the heads before it are evaluated and stored.  The output overwrites the checkpoint it was computed from,
// which is in shared memory by then; different heads never share bytes.
constexpr int DQ_THREADS = NT_LA + 32;
// A stage: the checkpoint, the KDA decay row, and -- for a head with at most DQ_ROWS live window entries, the case right
// after a prefill -- its window weights and its live rows of keys, values and (KDA) per-step decays.
constexpr int DQ_ROWS = 8;
__host__ __device__ constexpr int dq_off_w(int R) { return ck_bytes(R) + 512; }
__host__ __device__ constexpr int dq_off_rows(int R) { return dq_off_w(R) + 256; }
__host__ __device__ constexpr int dq_stage_bytes(int R) { return (dq_off_rows(R) + 3 * DQ_ROWS * 256 + 127) & ~127; }
struct DqInfo { int slot, h; float p; int valid; };
template <int R>
__global__ void __launch_bounds__(DQ_THREADS, 2)
dequant_kernel(lq_dims d, char* __restrict__ ssm, const uint16_t* __restrict__ Kbuf, const uint16_t* __restrict__ Ubuf,
               float* __restrict__ Wbuf, float* __restrict__ Pbuf, const uint16_t* __restrict__ Gbuf,
               int32_t* __restrict__ hcnt, const int32_t* __restrict__ idx, int nheads, int kda) {
    constexpr int KT = (3 * R + 15) / 16 * 16;            // K of the rank-R product: three pieces of R, padded to the instruction
    constexpr int KS = KT + 8;                            // row stride of the operands in bf16 elements (16 bytes of padding)
    constexpr int STAGE = dq_stage_bytes(R);
    extern __shared__ __align__(128) char dq_smem[];
    float* skq = reinterpret_cast<float*>(dq_smem + 2 * STAGE);   // [128] Sk / 127 (KDA: times pc)
    float* svp = skq + 128;                               // [128] Sv p
    uint16_t* Aop = reinterpret_cast<uint16_t*>(svp + 128);   // [128 rows v][KS]: Qp head | Qp remainder | Qp head | 0
    uint16_t* Bop = Aop + 128 * KS;                       // [128 cols c][KS]: Uc head | Uc head | Uc remainder | 0
    float* ws = reinterpret_cast<float*>(Bop + 128 * KS); // [64] window weights
    uint64_t* full = reinterpret_cast<uint64_t*>(ws + 64);    // [2] stage filled; [2] stage read to the end
    uint64_t* empty = full + 2;
    DqInfo* info = reinterpret_cast<DqInfo*>(empty + 2);  // [2]
    volatile int* okflag = reinterpret_cast<volatile int*>(info + 2);
    float* Kf = reinterpret_cast<float*>(info + 2) + 4;   // keys [Lp][WST] bf16 (columns permuted), values [Lp][WST] bf16; KDA: the keys are
                                                          // the head of k_j D_j, followed by its remainder [Lp][WST] and the raw keys [Lp][128]
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    constexpr int WST = 136;                              // GDN window rows in shared memory: 128 bf16 + 16 bytes, so that the
                                                          // eight rows of an ldmatrix tile fall into different bank groups
    const int Lp = (d.L + 15) & ~15;
    uint16_t* Ks = reinterpret_cast<uint16_t*>(Kf);       // keys: within every 16 columns c -> 8 (c % 4 / 2) + 2 (c / 4) + c % 2
    uint16_t* Us = Ks + Lp * WST;                         // values as stored
    uint16_t* Kl = Us + Lp * WST;                         // KDA: remainder of k_j D_j, same layout as Ks
    uint16_t* Kraw = Kl + Lp * WST;                       // KDA: keys as stored [Lp][128], read by the scan below

    if (tid == 0) {
        mbar_init(full + 0, 1); mbar_init(full + 1, 1);
        mbar_init(empty + 0, NT_LA / 32); mbar_init(empty + 1, NT_LA / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    __syncthreads();
    const int first = blockIdx.x, stride = gridDim.x;

    if (warp == NT_LA / 32) {
        // ================= the warp that runs ahead =================
        int l_slot = 0, l_h = 0, l_valid = 0;
        float l_p = 1.f;
        for (int i = 0; first + i * stride < nheads; ++i) {
            if ((i & 31) == 0) {                          // the scalars of the next 32 heads of this CTA, one head per lane
                const int pg = first + (i + lane) * stride;
                l_slot = 0; l_h = 0; l_valid = 0; l_p = 1.f;
                if (pg < nheads) {
                    const int hvv = pg % d.HV;
                    l_slot = idx[pg / d.HV];
                    l_valid = l_slot > 0 && l_slot < d.NS;
                    if (l_valid) {
                        const int64_t sh = int64_t(l_slot) * d.HV + hvv;
                        l_h = min(max(hcnt[sh], 0), d.L);
                        l_p = kda ? 1.f : Pbuf[sh];
                    }
                }
            }
            const int s = i & 1;
            if (i >= 2 && !warp_wait_bounded(empty + s, uint32_t((i >> 1) - 1) & 1u)) {
                if (lane == 0) atomicOr(&g_status, ST_PRODUCER_TIMEOUT);
                return;
            }
            const int src = i & 31;
            const int slot = __shfl_sync(0xffffffffu, l_slot, src), h = __shfl_sync(0xffffffffu, l_h, src);
            const int valid = __shfl_sync(0xffffffffu, l_valid, src);
            const float pp = __shfl_sync(0xffffffffu, l_p, src);
            if (lane == 0) {
                const int pg = first + i * stride, hv = pg % d.HV;
                info[s].slot = slot; info[s].h = h; info[s].p = pp; info[s].valid = valid;
                if (valid) {
                    fence_async_smem();                   // the stage's last readers used ordinary loads
                    const int64_t sh = int64_t(slot) * d.HV + hv;
                    const bool rows_in = h > 0 && h <= DQ_ROWS && d.L <= 64 && (d.L & 3) == 0;
                    const uint32_t rb = rows_in ? uint32_t(h) * 256u : 0u;
                    mbar_arrive_expect_tx(full + s, uint32_t(ck_bytes(R)) + (kda ? 512u : 0u) + (rows_in ? uint32_t(d.L) * 4u : 0u) + (kda ? 3u : 2u) * rb);
                    char* stg = dq_smem + s * STAGE;
                    bulk_g2s(stg, head_base(ssm, d.SS, slot, hv), uint32_t(ck_bytes(R)), full + s);
                    if (kda) bulk_g2s(stg + ck_bytes(R), Pbuf + sh * KD, 512u, full + s);
                    if (rows_in) {
                        bulk_g2s(stg + dq_off_w(R), Wbuf + sh * d.L, uint32_t(d.L) * 4u, full + s);
                        bulk_g2s(stg + dq_off_rows(R), Kbuf + sh * d.L * KD, rb, full + s);
                        bulk_g2s(stg + dq_off_rows(R) + DQ_ROWS * 256, Ubuf + sh * d.L * VD, rb, full + s);
                        if (kda) bulk_g2s(stg + dq_off_rows(R) + 2 * DQ_ROWS * 256, Gbuf + sh * d.L * KD, rb, full + s);
                    }
                } else {
                    mbar_arrive(full + s);                // padding row or null slot: nothing to fetch
                }
            }
            __syncwarp();
        }
        return;
    }

    // ================= the eight warps that evaluate and store =================
    for (int i = 0; first + i * stride < nheads; ++i) {
    const int s = i & 1;
    if (warp == 0) {
        const bool got = warp_wait_bounded(full + s, uint32_t(i >> 1) & 1u);
        if (lane == 0) *okflag = got ? 1 : 0;
    }
    named_bar(1, NT_LA);                                  // (also: every warp is done with the previous head's operands and window rows)
    if (*okflag == 0) {
        if (tid == 0) atomicOr(&g_status, ST_CONSUMER_TIMEOUT);
        return;
    }
    const DqInfo hi = info[s];
    if (!hi.valid) {
        if (lane == 0) mbar_arrive(empty + s);
        continue;
    }
    const int pg = first + i * stride;
    const int hv = pg % d.HV, slot = hi.slot, h = hi.h;
    const float p = hi.p;
    char* base = head_base(ssm, d.SS, slot, hv);
    const char* stg = dq_smem + s * STAGE;
    const uint32_t* cw = reinterpret_cast<const uint32_t*>(stg + CK_CODES);      // [128][32] code words
    const int64_t sh = int64_t(slot) * d.HV + hv;

    if (tid < 128) {
        const float pc = kda ? expf(reinterpret_cast<const float*>(stg + ck_bytes(R))[tid]) : 1.f;
        skq[tid] = reinterpret_cast<const float*>(stg + CK_SK)[tid] / QMAX * pc;
        svp[tid] = reinterpret_cast<const float*>(stg + CK_SV)[tid] * p;
        const uint16_t* uq = reinterpret_cast<const uint16_t*>(stg + CK_UQ);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float u = f16_to_f(uq[r * (KD + VD) + tid]) * pc, q = f16_to_f(uq[r * (KD + VD) + KD + tid]) * p;
            const uint16_t uh = f_to_bf16(u), qh = f_to_bf16(q);
            const uint16_t ul = f_to_bf16(u - bf16_to_f(uh)), ql = f_to_bf16(q - bf16_to_f(qh));
            Aop[tid * KS + r] = qh; Aop[tid * KS + R + r] = ql; Aop[tid * KS + 2 * R + r] = qh;
            Bop[tid * KS + r] = uh; Bop[tid * KS + R + r] = uh; Bop[tid * KS + 2 * R + r] = ul;
        }
#pragma unroll
        for (int r = 3 * R; r < KT; ++r) { Aop[tid * KS + r] = 0; Bop[tid * KS + r] = 0; }
    }
    // a short window came with the stage; a longer one is read from global memory here, four 16-byte pieces per thread in
    // flight at a time
    const bool rows_in = h > 0 && h <= DQ_ROWS && d.L <= 64 && (d.L & 3) == 0;
    if (tid < 64) {                                           // (all 64: the tensor-core window term reads whole steps of 16)
        float wv = 0.f;
        if (tid < h) wv = rows_in ? reinterpret_cast<const float*>(stg + dq_off_w(R))[tid] : Wbuf[sh * d.L + tid];
        ws[tid] = wv;
    }
    {
        const int hp = (h + 15) & ~15;                       // whole k-steps of 16 rows, the rows past h zero
        auto place = [&](int i2, const uint4& uv, const uint4& kv) {
            const int j = i2 >> 4, c8 = i2 & 15;              // row, 16-byte chunk (8 columns) of the row
            *reinterpret_cast<uint4*>(Us + j * WST + 8 * c8) = uv;
            if (kda) {
                reinterpret_cast<uint4*>(Kraw)[i2] = kv;
            } else {
                // the chunk holds columns 4 t .. 4 t + 7 of a group of 16 (t = 0 or 2): pairs (4t, 4t+1), (4t+4, 4t+5) go to the
                // first n-tile of the group at 2 t, 2 t + 2, pairs (4t+2, 4t+3), (4t+6, 4t+7) to the second at 8 + 2 t, 8 + 2 t + 2
                uint16_t* kd = Ks + j * WST + 16 * (c8 >> 1) + 4 * (c8 & 1);
                *reinterpret_cast<uint2*>(kd) = make_uint2(kv.x, kv.z);
                *reinterpret_cast<uint2*>(kd + 8) = make_uint2(kv.y, kv.w);
            }
        };
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        if (rows_in) {
            const uint4* kb = reinterpret_cast<const uint4*>(stg + dq_off_rows(R));
            const uint4* ub = reinterpret_cast<const uint4*>(stg + dq_off_rows(R) + DQ_ROWS * 256);
            for (int i2 = tid; i2 < hp * 16; i2 += NT_LA) {
                const bool live = (i2 >> 4) < h;
                place(i2, live ? ub[i2] : z, live ? kb[i2] : z);
            }
        } else if (h > 0) {
            const uint4* kb = reinterpret_cast<const uint4*>(Kbuf + sh * d.L * KD);
            const uint4* ub = reinterpret_cast<const uint4*>(Ubuf + sh * d.L * VD);
            for (int i0 = tid; i0 < hp * 16; i0 += 4 * NT_LA) {
                uint4 uv[4], kv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i2 = i0 + u * NT_LA;
                    const bool live = (i2 >> 4) < h;
                    uv[u] = live ? ldg_stream(ub + i2) : z;
                    kv[u] = live ? ldg_stream(kb + i2) : z;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i0 + u * NT_LA < hp * 16) place(i0 + u * NT_LA, uv[u], kv[u]);
            }
        }
    }
    named_bar(1, NT_LA);
    if (kda && h > 0) {
        if (tid < 128) {                       // D_j = prod_{j < i < h} e_i, backward running product per column; k_j D_j as a
            float dcur = 1.f;                  // bf16 head and remainder at the column's place in the permuted rows
            const int hp = (h + 15) & ~15;
            const int cp = (tid & ~15) + 8 * ((tid & 3) >> 1) + 2 * ((tid & 15) >> 2) + (tid & 1);
            for (int j = hp - 1; j >= h; --j) { Ks[j * WST + cp] = 0; Kl[j * WST + cp] = 0; }
            auto scan = [&](int j, float e) {
                const float kd = bf16_to_f(Kraw[j * 128 + tid]) * dcur;
                const uint16_t kh = f_to_bf16(kd);
                Ks[j * WST + cp] = kh;
                Kl[j * WST + cp] = f_to_bf16(kd - bf16_to_f(kh));
                dcur *= e;
            };
            if (rows_in) {
                const uint16_t* gs = reinterpret_cast<const uint16_t*>(stg + dq_off_rows(R) + 2 * DQ_ROWS * 256);
                for (int j = h - 1; j >= 0; --j) scan(j, f16_to_f(gs[j * KD + tid]));
            } else {                           // the per-step decays from global memory, eight in flight
                const uint16_t* gg = Gbuf + sh * d.L * KD + tid;
                for (int j0 = h - 1; j0 >= 0; j0 -= 8) {
                    uint16_t e[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) e[u] = j0 - u >= 0 ? __ldg(gg + (j0 - u) * KD) : uint16_t(0);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (j0 - u >= 0) scan(j0 - u, f16_to_f(e[u]));
                }
            }
        }
        named_bar(1, NT_LA);
    }

    const int r0 = 16 * warp + gid, r1 = r0 + 8;
    // rank-R term: A fragments of this warp's 16 rows once per K step, B fragments per n-tile
    uint32_t af[KT / 16][4];
#pragma unroll
    for (int ks = 0; ks < KT / 16; ++ks) {
        af[ks][0] = *reinterpret_cast<const uint32_t*>(Aop + r0 * KS + 16 * ks + 2 * tig);
        af[ks][1] = *reinterpret_cast<const uint32_t*>(Aop + r1 * KS + 16 * ks + 2 * tig);
        af[ks][2] = *reinterpret_cast<const uint32_t*>(Aop + r0 * KS + 16 * ks + 8 + 2 * tig);
        af[ks][3] = *reinterpret_cast<const uint32_t*>(Aop + r1 * KS + 16 * ks + 8 + 2 * tig);
    }
    const int cn = 4 * (gid >> 1) + (gid & 1);              // column (within a group of 16) that n index gid of the first n-tile stands for
    const float sv0 = svp[r0], sv1 = svp[r1];
    float* out = reinterpret_cast<float*>(base);            // (everything of the slot that is read was copied to shared memory above)
    // two groups of 16 columns at a time, start to finish: sixteen accumulators per thread instead of sixty-four, and the
    // values of a window entry are fetched four times per entry, not eight
#pragma unroll 1
    for (int qp = 0; qp < 4; ++qp) {
        float a0[2][4], a1[2][4];                           // [group][column]: rows r0 and r1, columns 16 q + 4 tig + k
#pragma unroll
        for (int g2 = 0; g2 < 2; ++g2) {
            const int q = 2 * qp + g2;
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < KT / 16; ++ks) {
                const uint16_t* b0p = Bop + (16 * q + cn) * KS + 16 * ks + 2 * tig;
                const uint16_t* b1p = b0p + 2 * KS;
                mma_bf16_16816(c0, af[ks][0], af[ks][1], af[ks][2], af[ks][3], *reinterpret_cast<const uint32_t*>(b0p),
                               *reinterpret_cast<const uint32_t*>(b0p + 8));
                mma_bf16_16816(c1, af[ks][0], af[ks][1], af[ks][2], af[ks][3], *reinterpret_cast<const uint32_t*>(b1p),
                               *reinterpret_cast<const uint32_t*>(b1p + 8));
            }
            // codes: one word = this lane's four columns of a row
            // (packed pairs: the same three roundings per element -- convert, times the column scale, fused with the row
            //  scale into the rank-R term -- in half the instructions)
            const float4 sk4 = *reinterpret_cast<const float4*>(skq + 16 * q + 4 * tig);
            const float2 sk01 = make_float2(sk4.x, sk4.y), sk23 = make_float2(sk4.z, sk4.w);
            const float2 s0 = make_float2(sv0, sv0), s1 = make_float2(sv1, sv1);
            float2 f01, f23, g01, g23;
            s8x4_to_f2x2(cw[r0 * 32 + 4 * q + tig], f01, f23);
            s8x4_to_f2x2(cw[r1 * 32 + 4 * q + tig], g01, g23);
            const float2 x01 = __ffma2_rn(__fmul2_rn(f01, sk01), s0, make_float2(c0[0], c0[1]));
            const float2 x23 = __ffma2_rn(__fmul2_rn(f23, sk23), s0, make_float2(c1[0], c1[1]));
            const float2 y01 = __ffma2_rn(__fmul2_rn(g01, sk01), s1, make_float2(c0[2], c0[3]));
            const float2 y23 = __ffma2_rn(__fmul2_rn(g23, sk23), s1, make_float2(c1[2], c1[3]));
            a0[g2][0] = x01.x; a0[g2][1] = x01.y; a0[g2][2] = x23.x; a0[g2][3] = x23.y;
            a1[g2][0] = y01.x; a1[g2][1] = y01.y; a1[g2][2] = y23.x; a1[g2][3] = y23.y;
        }
        // live window entries: sum_j (w_j u_j[v]) (k_j[c] D_j[c]) on the tensor cores, 16 entries per step.  A = the values, read
        // transposed from their rows ([j][v] -> rows v, K index j), scaled by w_j in registers and split into a bf16 head and
        // remainder; B = the keys, read transposed from their column-permuted rows (GDN: exact in bf16; KDA: head and remainder
        // of the decayed keys, three products).
        for (int j0 = 0; j0 < h; j0 += 16) {
            uint32_t au[4];
            ldmatrix_x4_trans(au, Us + (j0 + (lane & 7) + ((lane >> 4) << 3)) * WST + 16 * warp + (((lane >> 3) & 1) << 3));
            const float2 w01 = *reinterpret_cast<const float2*>(ws + j0 + 2 * tig), w89 = *reinterpret_cast<const float2*>(ws + j0 + 8 + 2 * tig);
            uint32_t ah[4], al[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {                    // au[0], au[1]: entries j0 + 2 tig, + 1; au[2], au[3]: j0 + 8 + 2 tig, + 1
                const float2 wv = i < 2 ? w01 : w89;
                const float2 uv = bf16x2_to_f2(au[i]);
                const float x0 = uv.x * wv.x, x1 = uv.y * wv.y;
                ah[i] = f2_to_bf16x2(x0, x1);
                const float2 hv2 = bf16x2_to_f2(ah[i]);
                al[i] = f2_to_bf16x2(x0 - hv2.x, x1 - hv2.y);
            }
#pragma unroll
            for (int g2 = 0; g2 < 2; ++g2) {
                const int koff = (j0 + (lane & 7) + (((lane >> 3) & 1) << 3)) * WST + 16 * (2 * qp + g2) + ((lane >> 4) << 3);
                uint32_t bk[4];                              // keys of the group's two n-tiles: (tile 0: rows j0.., j0 + 8..), (tile 1: ..)
                ldmatrix_x4_trans(bk, Ks + koff);
                float c0[4] = {a0[g2][0], a0[g2][1], a1[g2][0], a1[g2][1]}, c1[4] = {a0[g2][2], a0[g2][3], a1[g2][2], a1[g2][3]};
                mma_bf16_16816(c0, ah[0], ah[1], ah[2], ah[3], bk[0], bk[1]);
                mma_bf16_16816(c0, al[0], al[1], al[2], al[3], bk[0], bk[1]);
                mma_bf16_16816(c1, ah[0], ah[1], ah[2], ah[3], bk[2], bk[3]);
                mma_bf16_16816(c1, al[0], al[1], al[2], al[3], bk[2], bk[3]);
                if (kda) {
                    uint32_t bl[4];
                    ldmatrix_x4_trans(bl, Kl + koff);
                    mma_bf16_16816(c0, ah[0], ah[1], ah[2], ah[3], bl[0], bl[1]);
                    mma_bf16_16816(c1, ah[0], ah[1], ah[2], ah[3], bl[2], bl[3]);
                }
                a0[g2][0] = c0[0]; a0[g2][1] = c0[1]; a1[g2][0] = c0[2]; a1[g2][1] = c0[3];
                a0[g2][2] = c1[0]; a0[g2][3] = c1[1]; a1[g2][2] = c1[2]; a1[g2][3] = c1[3];
            }
        }
#pragma unroll
        for (int g2 = 0; g2 < 2; ++g2) {
            const int q = 2 * qp + g2;
            *reinterpret_cast<float4*>(out + r0 * KD + 16 * q + 4 * tig) = make_float4(a0[g2][0], a0[g2][1], a0[g2][2], a0[g2][3]);
            *reinterpret_cast<float4*>(out + r1 * KD + 16 * q + 4 * tig) = make_float4(a1[g2][0], a1[g2][1], a1[g2][2], a1[g2][3]);
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + s);                  // this warp has read the last of the stage
    if (!kda) {
        for (int j = tid; j < d.L; j += NT_LA) Wbuf[sh * d.L + j] = 0.f;
        if (tid == 0) {
            Pbuf[sh] = 1.f;
            hcnt[sh] = 0;
        }
    }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// low-rank factorisation of x [n][K][V]
// ------------------------------------------------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(NT_LA, 1)
lowrank_kernel(const float* __restrict__ x, const float* __restrict__ Q0, float* __restrict__ U, float* __restrict__ Q,
               int iters) {
    extern __shared__ __align__(16) float smem[];
    float* M = smem;                      // [K][LDB]: row = key index, column = value index
    float* Qs = M + 128 * LDB;            // [V][R]
    float* Ps = Qs + 128 * R;             // [K][R]
    float* scr = Ps + 128 * R;
    const int tid = threadIdx.x;
    const float* xb = x + int64_t(blockIdx.x) * KD * VD;
    for (int i = tid; i < 128 * 32; i += NT_LA) {
        const float4 v = reinterpret_cast<const float4*>(xb)[i];
        *reinterpret_cast<float4*>(M + (i >> 5) * LDB + (i & 31) * 4) = v;
    }
    for (int i = tid; i < 128 * R; i += NT_LA) Qs[i] = Q0[i];
    __syncthreads();
    for (int it = 0; it < iters; ++it) {
        rowdot<R>(M, Qs, Ps, scr, tid);       // P = x Q
        mgs_cols<R>(Ps, tid);
        coldot<R>(M, Ps, Qs, scr, tid);       // Q = x^T P
        mgs_cols<R>(Qs, tid);
    }
    rowdot<R>(M, Qs, Ps, scr, tid);           // U = x Q
    float* Ub = U + int64_t(blockIdx.x) * KD * R;
    float* Qb = Q + int64_t(blockIdx.x) * VD * R;
    for (int i = tid; i < 128 * R; i += NT_LA) {
        Ub[i] = Ps[i];
        Qb[i] = Qs[i];
    }
}

}  // namespace lq

using namespace lq;

extern "C" int lq_quantize(const lq_dims* d, void* ssm, float* Wbuf, float* Pbuf, void* Gbuf, int32_t* hcnt,
                           const float* Q0, const int32_t* idx, int32_t N, int32_t kda, int32_t iters, void* stream) {
    int rc = check_dims(d);
    if (rc) return rc;
    if (!ssm || !Wbuf || !Pbuf || !hcnt || !Q0 || (N > 0 && !idx) || (kda && !Gbuf)) return LQ_ERR_NULL;
    if (N < 0 || iters < 0) return LQ_ERR_RANGE;
    if (misaligned16({ssm}) || (kda && misaligned16({Gbuf}))) return LQ_ERR_ALIGN;
    if (N == 0) return LQ_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nheads = N * d->HV, cap = 2 * device_sm_count();
    dim3 grid(unsigned(nheads < cap ? nheads : cap)), block(NT_LA);
    if (d->R == 4) {
        if ((rc = ensure_smem((const void*)quantize_kernel<4>, qz_smem_bytes<4>()))) return rc;
        quantize_kernel<4><<<grid, block, qz_smem_bytes<4>(), st>>>(*d, (char*)ssm, Wbuf, Pbuf, (uint16_t*)Gbuf, hcnt, Q0, idx, nheads, kda, iters);
    } else {
        if ((rc = ensure_smem((const void*)quantize_kernel<8>, qz_smem_bytes<8>()))) return rc;
        quantize_kernel<8><<<grid, block, qz_smem_bytes<8>(), st>>>(*d, (char*)ssm, Wbuf, Pbuf, (uint16_t*)Gbuf, hcnt, Q0, idx, nheads, kda, iters);
    }
    return finish_launch();
}

extern "C" int lq_dequant(const lq_dims* d, void* ssm, const void* Kbuf, const void* Ubuf, float* Wbuf, float* Pbuf,
                          const void* Gbuf, int32_t* hcnt, const int32_t* idx, int32_t N, int32_t kda, void* stream) {
    int rc = check_dims(d);
    if (rc) return rc;
    if (!ssm || !Kbuf || !Ubuf || !Wbuf || !Pbuf || !hcnt || (N > 0 && !idx) || (kda && !Gbuf)) return LQ_ERR_NULL;
    if (N < 0) return LQ_ERR_RANGE;
    if (misaligned16({ssm, Kbuf, Ubuf})) return LQ_ERR_ALIGN;
    if (N == 0) return LQ_OK;
    // two checkpoint stages, folded scales, factors, weights, barriers, window rows (bf16; KDA: decayed keys as head and remainder)
    const int kt = (3 * d->R + 15) / 16 * 16 + 8;               // operand row of the rank-R product, bf16 elements
    const size_t win = size_t((d->L + 15) & ~15) * (kda ? 3 * 136 * 2 + 128 * 2 : 2 * 136 * 2);
    const size_t smem = size_t(2) * dq_stage_bytes(d->R) + sizeof(float) * (2 * 128 + 64) + size_t(2) * 128 * kt * 2 + 4 * sizeof(uint64_t) +
                        2 * sizeof(DqInfo) + 16 + win;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nheads = N * d->HV;
    const int cap = 2 * device_sm_count();
    dim3 grid(unsigned(nheads < cap ? nheads : cap)), block(DQ_THREADS);
    if (d->R == 4) {
        if ((rc = ensure_smem((const void*)dequant_kernel<4>, smem))) return rc;
        dequant_kernel<4><<<grid, block, smem, st>>>(*d, (char*)ssm, (const uint16_t*)Kbuf, (const uint16_t*)Ubuf, Wbuf, Pbuf,
                                                     (const uint16_t*)Gbuf, hcnt, idx, nheads, kda);
    } else {
        if ((rc = ensure_smem((const void*)dequant_kernel<8>, smem))) return rc;
        dequant_kernel<8><<<grid, block, smem, st>>>(*d, (char*)ssm, (const uint16_t*)Kbuf, (const uint16_t*)Ubuf, Wbuf, Pbuf,
                                                     (const uint16_t*)Gbuf, hcnt, idx, nheads, kda);
    }
    return finish_launch();
}

extern "C" int lq_lowrank(const float* x, const float* Q0, float* U, float* Q, int32_t n, int32_t K, int32_t V, int32_t r,
                          int32_t iters, void* stream) {
    if (!x || !Q0 || !U || !Q) return LQ_ERR_NULL;
    if (K != KD || V != VD || (r != 4 && r != 8)) return LQ_ERR_UNSUPPORTED;
    if (n < 0 || iters < 0) return LQ_ERR_RANGE;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return LQ_ERR_ALIGN;
    if (n == 0) return LQ_OK;
    const size_t smem = sizeof(float) * (128 * LDB + 3 * 128 * r);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc;
    if (r == 4) {
        if ((rc = ensure_smem((const void*)lowrank_kernel<4>, smem))) return rc;
        lowrank_kernel<4><<<n, NT_LA, smem, st>>>(x, Q0, U, Q, iters);
    } else {
        if ((rc = ensure_smem((const void*)lowrank_kernel<8>, smem))) return rc;
        lowrank_kernel<8><<<n, NT_LA, smem, st>>>(x, Q0, U, Q, iters);
    }
    return finish_launch();
}
