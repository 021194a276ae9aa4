// Search passes for grid sides d = N1 * N2 above the whole-line kernels' range
// (vesper_regpass.cuh): every line FFT runs as two register steps (of N1 and of
// N2 points), the steps of a line meeting in shared memory.
//
//   A  one x plane per CTA.  The CTA gathers the plane; each warp then owns tiles of
//      4 packed z lines (8 rows), which it transforms along z and unpacks into rows
//      with warp barriers only; then the block transforms the columns along y,
//      straight to S.
//   B  W spectrum columns per CTA, several rotations one after another: the
//      columns' target values stay in registers for all of them.
//   C  one x plane per CTA: inverse y in place, then each warp owns PL row
//      pairs for the inverse z transform and the argmax.
//
// Inputs, outputs and layouts are those of the radix-stage passes.  Two kinds of
// arithmetic: the radix-stage passes' own, bit for bit (the general form), or line
// DFTs whose coprime factors split without twiddles (PFA) with the inverse's
// steps in the opposite order.
//
// What bounds them (GB300, mode V, microseconds per rotation A / B / C, against
// the kernels they replace): side 75 2.57 / 1.56 / 0.91 (one block-wide step after
// another, general gather in line: 5.41 / 1.74 / 1.04), side 48 0.69 / 0.60 / 0.29
// (radix stages 2.26 / 1.60 / 1.06), side 80 2.82 / 2.20 / 1.16 (11.9 / 7.4 / 3.1),
// prob mode at side 64 3.4 / 2.6 / 1.17 (18.0 / 5.4 / 2.7).  A is bound by issue
// slots and the L1 data path together (68 % and 72 % at side 75, 73 % and 83 % at 48;
// one warp per tile gives 45 % of the warps): strides without bank conflicts took side
// 75 from 4.17 to 3.93, one warp per tile within 64 registers to 3.48, and the middle
// voxels of odd sides, loaded together and shared out over the CTA, to 3.14; prob mode
// at side 64 4.51 -> 3.97 with lines and columns that do not meet in a bank.  A query
// fills a ball of its grid, and the rotated one a ball too: leaving out the z steps,
// lines and planes outside it took side 75 from 3.14 to 2.50 and prob mode at side 64
// from 3.97 to 3.30 (a ball of 0.42 of the side).  C is bound
// by issue slots (72 %): one 32-bit comparison per voxel instead of a 64-bit key took
// side 75 from 0.98 to 0.87.  B is
// bound by the S and T it reads: T from L2 once per 8 rotations instead of once
// each took side 75 from 1.74 to 1.52.
#pragma once

#include "vesper_regfft.cuh"
#include "vesper_tilegather.cuh"

namespace vg {

// Shared-memory layout of a plane.  A 64-bit access is conflict-free when the 16
// lanes of a half warp fall in 16 different 8-byte banks.  With the row stride RS
// = 2 mod 4, four consecutive packed lines (stride LS = 2 RS) start 4 banks
// apart, so lanes that run over 4 lines and then over 4 consecutive elements cover
// all 16; between the steps element (k1, j2) of a line sits at P2 k1 + j2 with P2
// odd, so that runs over k1 do the same; CS = N2 mod 4 continues the pattern
// from one channel to the next (2 where N2 is a multiple of 4: runs over 8 lines of
// two channels).
constexpr int up_to_mod(int n, int mod, int rem) { return n + ((rem - n) % mod + mod) % mod; }
// SPLIT: a line's elements lie half in its first row's storage, half in its second's.
template <int N1, int N2, bool SPLIT = false>
struct TGeom {
    static constexpr int D = N1 * N2, H = D / 2 + 1, NP = (D + 1) / 2;
    static constexpr int P2 = N2 | 1;
    static constexpr int kHalf = SPLIT ? (N1 + 1) / 2 * P2 : (N1 * P2 + 1) / 2;
    static constexpr int RS = up_to_mod(H > kHalf ? H : kHalf, 4, 2);   // row stride
    static constexpr int LS = 2 * RS;          // packed line p lives in rows 2p and 2p + 1
    static constexpr int CS = up_to_mod(NP * LS, 4, N2 % 4 ? N2 % 4 : 2);   // channel stride
    static constexpr int TP = (NP + 3) / 4;    // gather tiles of 4 lines
    // where element z = j2 + N2 j1 of a line waits for step 1
    static __device__ __forceinline__ int pos(int z) { return P2 == N2 ? z : z / N2 * P2 + z % N2; }
};

// Column kz and row of item t of a step along y in shared memory: a half warp stays in one
// row as long as that leaves no lane idle (runs over whole rows of H put two rows into
// most half warps, whose banks overlap), the columns past the last 16 of each row follow.
template <int H> __device__ __forceinline__ void column_item(int t, int rows, int &kz, int &row) {
    constexpr int HM = H / 16 * 16, HR = H - HM;
    const int u = t - rows * HM;
    if (HM && u < 0) {
        row = t / (HM ? HM : 1);
        kz = t - row * HM;
    } else {
        row = u / (HR ? HR : 1);
        kz = HM + u - row * HR;
    }
}

// ---- pass A -------------------------------------------------------------------
// Lines per round of the second z step: as many as the warp's lanes hold, whole groups
// of 4 (which fall in different banks) where that costs no round.
__host__ __device__ constexpr int lines_per_round(int items, int lines) {
    const int most = 32 / items < lines ? 32 / items : lines, four = most / 4 * 4;
    return four && (lines + four - 1) / four == (lines + most - 1) / most ? four : most;
}
template <int SRC, int N1, int N2>
__host__ __device__ constexpr size_t smem_ta() {
    using G = TGeom<N1, N2>;
    return (size_t)((G::D + 1) / 2 * 2) * sizeof(float2) + (size_t)src_nch<SRC>() * G::CS * sizeof(float2);
}

// Warps per CTA: one per 4-line tile.  Resident CTAs the register budget is
// sized for: as many as shared memory allows, with at least 64 registers a thread.
template <int N1, int N2> __host__ __device__ constexpr int ta_warps() { return TGeom<N1, N2>::TP; }
template <int SRC, int N1, int N2> __host__ __device__ constexpr int ta_ctas() {
    constexpr int by_smem = (int)((228 * 1024) / (smem_ta<SRC, N1, N2>() + 1024));
    constexpr int by_regs = 65536 / (64 * ta_warps<N1, N2>() * 32);
    return by_smem < by_regs ? by_smem : by_regs;
}

template <int SRC, int N1, int N2, bool PFA>
__device__ __forceinline__ void tpass_a(const PassA2 &a, int c0) {
    using G = TGeom<N1, N2>;
    constexpr int D = G::D, H = G::H, NP = G::NP, RS = G::RS, LS = G::LS, CS = G::CS, P2 = G::P2, NCH = src_nch<SRC>();
    constexpr int NW = ta_warps<N1, N2>();
    extern __shared__ __align__(16) unsigned char smem[];
    const int x = blockIdx.x, b = blockIdx.y, r = a.r0 + b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2 *twn = (float2 *)smem;
    float2 *buf = twn + (D + 1) / 2 * 2;   // [NCH][NP][LS]
    twiddles_n(D, twn);
    if (x == 0 && c0 == 0 && threadIdx.x < a.nscore) a.keys[(size_t)r * a.nscore + threadIdx.x] = 0ull;
    float F[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) F[i] = __ldg(a.rotmats + (size_t)r * 9 + i);
    static_assert(NW == G::TP, "one tile per warp");
    const bool empty = gather_planes<SRC, D, LS, CS, NW, true>(a, F, b, x, 1, buf, [](int z) { return G::pos(z); });
    __syncthreads();
    const int pt = warp;
    if (empty) {   // zeros transform to zeros
        for (int l = 0; l < 4 && pt * 4 + l < NP; ++l)
#pragma unroll
            for (int c = 0; c < NCH; ++c)
                for (int k = lane; k < LS; k += 32) buf[c * CS + (pt * 4 + l) * LS + k] = make_float2(0.f, 0.f);
    } else {
        // z step 1, in place: items (c, j2, line), line fastest
        for (int it = lane; it < NCH * 4 * N2; it += 32) {
            const int p = pt * 4 + (it & 3), j2 = (it >> 2) % N2, c = (it >> 2) / N2;
            if (p < NP) {
                float2 *line = buf + c * CS + p * LS + j2;
                float2 v[N1];
#pragma unroll
                for (int j1 = 0; j1 < N1; ++j1) v[j1] = line[P2 * j1];
                line_dft<N1, D, false, PFA>(v, twn);
#pragma unroll
                for (int k1 = 0; k1 < N1; ++k1) line[P2 * k1] = (k1 && j2) ? step_twiddle<false, PFA>(v[k1], twn[j2 * k1]) : v[k1];
            }
        }
        __syncwarp();
        // z step 2 and unpack into the line's own two rows: items (line, q) of k1 = q and its
        // mirror N1 - q (q = 0: 0 and, N1 even, N1 / 2, which mirror themselves), whole
        // lines per round, read before they are written
        constexpr bool EV = N1 % 2 == 0;
        constexpr int NQ = (N1 + 1) / 2, LPR = lines_per_round(NQ, NCH * 4);
        const int lq = lane % LPR, q = lane / LPR, q2 = q ? N1 - q : EV ? N1 / 2 : 0;   // line fastest
#pragma unroll 1
        for (int l0 = 0; l0 < NCH * 4; l0 += LPR) {
            const int l = l0 + lq, p = pt * 4 + (l & 3), c = l >> 2;
            const bool on = q < NQ && l < NCH * 4 && p < NP;
            float2 *line = buf + c * CS + p * LS;
            float2 u[N2], w2[N2];
            if (on) {
#pragma unroll
                for (int j2 = 0; j2 < N2; ++j2) u[j2] = line[P2 * q + j2];
#pragma unroll
                for (int j2 = 0; j2 < N2; ++j2) w2[j2] = line[P2 * q2 + j2];
                line_dft<N2, D, false, PFA>(u, twn);
                line_dft<N2, D, false, PFA>(w2, twn);
            }
            __syncwarp();
            if (on) {
                float2 *row0 = line, *row1 = line + RS;
#pragma unroll
                for (int k2 = 0; k2 < N2; ++k2) {
                    const int k = q + N1 * k2;
                    if (k < H) {
                        float2 A, B;
                        unpack_pair(u[k2], (q == 0) ? u[(N2 - k2) % N2] : w2[N2 - 1 - k2], A, B);
                        row0[k] = A;
                        row1[k] = B;
                    }
                    const int kb = q2 + N1 * k2;
                    if ((EV || q != 0) && kb < H) {
                        float2 A, B;
                        unpack_pair(w2[k2], (q == 0) ? w2[N2 - 1 - k2] : u[N2 - 1 - k2], A, B);
                        row0[kb] = A;
                        row1[kb] = B;
                    }
                }
            }
        }
    }
    float2 *out = a.S + (((size_t)b * a.nch + c0) * D + x) * (size_t)(D * H);
    if (!__syncthreads_or(!empty)) {   // no value on the whole plane
        for (int c = 0; c < NCH; ++c)
            for (int e = threadIdx.x; e < D * H; e += NW * 32) out[(size_t)c * (D * D * H) + e] = make_float2(0.f, 0.f);
        return;
    }
    // y step 1, in place: items (c, j2, kz), kz fastest
    for (int t = threadIdx.x; t < NCH * N2 * H; t += NW * 32) {
        int kz, cj;
        column_item<H>(t, NCH * N2, kz, cj);
        const int j2 = cj % N2, c = cj / N2;
        float2 *col = buf + c * CS + j2 * RS + kz;
        float2 v[N1];
#pragma unroll
        for (int j1 = 0; j1 < N1; ++j1) v[j1] = col[N2 * j1 * RS];
        line_dft<N1, D, false, PFA>(v, twn);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) col[N2 * k1 * RS] = (k1 && j2) ? step_twiddle<false, PFA>(v[k1], twn[j2 * k1]) : v[k1];
    }
    __syncthreads();
    // y step 2: items (c, k1, kz), kz fastest -> S rows ky = k1 + N1 k2
    for (int t = threadIdx.x; t < NCH * N1 * H; t += NW * 32) {
        const int kz = t % H, ck = t / H, k1 = ck % N1, c = ck / N1;
        const float2 *col = buf + c * CS + N2 * k1 * RS + kz;
        float2 u[N2];
#pragma unroll
        for (int j2 = 0; j2 < N2; ++j2) u[j2] = col[j2 * RS];
        line_dft<N2, D, false, PFA>(u, twn);
        float2 *dst = out + (size_t)c * (D * D * H) + k1 * H + kz;
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) dst[N1 * k2 * H] = u[k2];
    }
}

template <int SRC, int N1, int N2, bool PFA>
__global__ void __launch_bounds__(ta_warps<N1, N2>() * 32, ta_ctas<SRC, N1, N2>()) k_tpass_a(const PassA2 a) {
    tpass_a<SRC, N1, N2, PFA>(a, 0);
}
// prob mode: the vector channels and the probability channels in CTAs of their own
template <int N1, int N2, bool PFA>
__global__ void __launch_bounds__(ta_warps<N1, N2>() * 32, ta_ctas<kSrcProb, N1, N2>()) k_tpass_a_prob(const PassA2 a) {
    if (blockIdx.z == 0)
        tpass_a<kSrcVec, N1, N2, PFA>(a, 0);
    else
        tpass_a<kSrcProb, N1, N2, PFA>(a, 3);
}

// ---- pass B -------------------------------------------------------------------
// Columns and threads per CTA, rotations side by side in it, CTAs that registers are
// budgeted for.  The steps of N1 points have N2 items per column, channel and rotation,
// those of N2 points N1, and every step ends at a barrier, so a shape leaves threads
// idle (a step costs its rounds times its points); shared memory and registers (target
// values, and a line of either step) decide how many CTAs cover one another's barriers.
// The measured rates of 90 pairs of shapes go as busy^0.4 warps^0.36 CTAs^0.14, hence
// the cubes; a shape other than a thread per item of the second forward step is taken
// where that promises a tenth (a sixth for one channel, whose three rotations already
// share the barriers: below that 42 and 100 lost), and never for PFA sides, which have
// no fourth step (side 75: 1.5 to 1.6 either way).  Microseconds per rotation, a thread per
// item before and after: mode V 48 0.69 -> 0.61, 54 1.18 -> 0.94, 72 4.19 -> 2.33,
// 81 5.57 -> 3.16, 88 5.89 -> 3.88, 91 6.81 -> 4.37, 96 9.08 -> 6.30; one channel 39
// 0.27 -> 0.18, 66 0.96 -> 0.65, 78 2.44 -> 1.13, 96 4.01 -> 2.01; prob mode 48 1.65 ->
// 1.18, 72 8.8 -> 4.2, 78 12.2 -> 7.3, 96 19.0 -> 12.2.
struct BShape {
    int cols, side, threads, ctas;
    double rank;
};
__host__ __device__ constexpr BShape tb_rank(int nch, int n1, int n2, int w, int nr, int t) {
    const int its = (n1 * w + t - 1) / t, d = n1 * n2;
    const int sm = nr * (nch + 1) * d * w * 8 + d * 8 + 1024;
    const int held = 2 * its * nch * n2 + (n1 > 2 * n2 ? 2 * n1 : 4 * n2) + 32;
    const int regs = held < 64 ? 64 : held > 255 ? 255 : (held + 7) / 8 * 8;
    const int by_smem = 228 * 1024 / sm, by_regs = 65536 / (regs * t);
    const int ctas = by_smem < by_regs ? by_smem : by_regs;
    if (ctas < 1 || held > 200) return BShape{w, nr, t, 1, 0.0};
    const double cost = (double)t * ((nr * nch * n2 * w + t - 1) / t * n1 + its * nr * nch * n2 +
                                     (nr * n2 * w + t - 1) / t * n1 + its * nr * n2);
    const double busy = nr * (double)(2 * nch + 2) * d * w / cost;
    const double warps = ctas * t / 32 < 24 ? ctas * t / 32.0 : 24.0;
    return BShape{w, nr, t, ctas, busy * busy * busy * warps * warps * warps * (ctas < 4 ? ctas : 4)};
}
template <int NCH, int N1, int N2, bool PFA>
__host__ __device__ constexpr BShape tb_shape() {
    constexpr int w0 = N1 >= 9 ? 16 : 32;
    BShape best = tb_rank(NCH, N1, N2, w0, NCH == 1 ? 3 : 1, (N1 * w0 + 31) / 32 * 32);
    best.ctas = 0;   // no budget
    if (PFA) return best;
    double least = (NCH == 1 ? 3.51 : 2.14) * best.rank;   // 1.17^8, 1.1^8
    for (int w = 16; w <= 32; w += 16)
        for (int nr = 1; nr <= 4; ++nr)
            for (int t = 64; t <= 512; t += 32) {
                const BShape s = tb_rank(NCH, N1, N2, w, nr, t);
                if (s.rank > least) {
                    best = s;
                    least = 1.0001 * s.rank;
                }
            }
    return best;
}
// SH: the channels that the shape is chosen for (prob mode's two kinds share a launch)
template <int SH, int N1, int N2, bool PFA>
__host__ __device__ constexpr size_t smem_tb() {
    constexpr BShape s = tb_shape<SH, N1, N2, PFA>();
    return (size_t)((N1 * N2 + 1) / 2 * 2) * sizeof(float2) +
           (size_t)s.side * (SH + 1) * N1 * N2 * s.cols * sizeof(float2);
}

template <int NCH, int SH, int N1, int N2, bool PFA>
__device__ __forceinline__ void tpass_b(const PassB2 &a, int c0, int grp, int nb, int rper) {
    constexpr BShape shape = tb_shape<SH, N1, N2, PFA>();
    constexpr int D = N1 * N2, H = D / 2 + 1, dH = D * H, W = shape.cols, TB = shape.threads, NR = shape.side;
    constexpr int IT = (N1 * W + TB - 1) / TB;   // items of step 2 per thread
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *twn = (float2 *)smem;
    float2 *buf = twn + (D + 1) / 2 * 2;              // [NR][NCH][D][W]
    float2 *pbuf = buf + (size_t)NR * NCH * D * W;    // [NR][D][W]
    const int j0 = blockIdx.x * W, b0 = blockIdx.y * rper, b1 = min(nb, b0 + rper);
    twiddles_n(D, twn);
    // the thread's target values: items (k1, w) of step 2, for every rotation
    float2 tv[IT][NCH][N2];
#pragma unroll
    for (int i = 0; i < IT; ++i) {
        const int t = threadIdx.x + i * TB, w = t % W, k1 = t / W;
        const bool on = t < N1 * W && j0 + w < dH;
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2)
                tv[i][c][k2] = on ? __ldg(a.T + (size_t)(c0 + c) * D * dH + (size_t)(k1 + N1 * k2) * dH + j0 + w)
                                  : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int b = b0; b < b1; b += NR) {
        const float2 *src = a.S + ((size_t)b * a.nch + c0) * D * dH + j0;
        // forward step 1: items (rotation, c, j2, w) from global
        for (int t = threadIdx.x; t < NR * NCH * N2 * W; t += TB) {
            const int w = t % W, cj = t / W, j2 = cj % N2, rc = cj / N2, c = rc % NCH, rr = rc / NCH;
            float2 v[N1];
            const float2 *s = src + ((size_t)(rr * a.nch + c) * D + j2) * dH + w;
            const bool on = j0 + w < dH && (NR == 1 || b + rr < b1);
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) v[j1] = on ? s[(size_t)(N2 * j1) * dH] : make_float2(0.f, 0.f);
            line_dft<N1, D, false, PFA>(v, twn);
            float2 *col = buf + (size_t)(rc * D + j2) * W + w;
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) col[N2 * k1 * W] = (k1 && j2) ? step_twiddle<false, PFA>(v[k1], twn[j2 * k1]) : v[k1];
        }
        __syncthreads();
        // forward step 2, product with conj(T), channel sum; PFA: inverse step 2 with
        // conjugate twiddles into pbuf rows k1 + N1 j2, else the sums themselves there
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int t = threadIdx.x + i * TB, w = t % W, k1 = t / W;
            if (t < N1 * W) {
#pragma unroll
                for (int rr = 0; rr < NR; ++rr) {
                    float2 acc[N2];
#pragma unroll
                    for (int k2 = 0; k2 < N2; ++k2) acc[k2] = make_float2(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < NCH; ++c) {
                        const float2 *col = buf + (size_t)((rr * NCH + c) * D + N2 * k1) * W + w;
                        float2 u[N2];
#pragma unroll
                        for (int j2 = 0; j2 < N2; ++j2) u[j2] = col[j2 * W];
                        line_dft<N2, D, false, PFA>(u, twn);
#pragma unroll
                        for (int k2 = 0; k2 < N2; ++k2) acc[k2] = cadd(acc[k2], cmul(tv[i][c][k2], u[k2]));
                    }
                    if constexpr (PFA) rdft<N2, true>(acc);
                    float2 *col = pbuf + (rr * D + k1) * W + w;
#pragma unroll
                    for (int j2 = 0; j2 < N2; ++j2)
                        col[N1 * j2 * W] = (PFA && k1 && j2) ? cmulc(acc[j2], twn[j2 * k1]) : acc[j2];
                }
            }
        }
        __syncthreads();
        float2 *dst = a.U + ((size_t)b * a.ngrp + grp) * D * dH + j0;
        if constexpr (!PFA) {
            // inverse steps in the forward's order: step 1 in place, items (rotation,
            // j2, w); step 2, items (rotation, k1, w) -> U rows x = k1 + N1 k2
            for (int t = threadIdx.x; t < NR * N2 * W; t += TB) {
                const int w = t % W, rj = t / W, j2 = rj % N2, rr = rj / N2;
                float2 *col = pbuf + (rr * D + j2) * W + w;
                float2 v[N1];
#pragma unroll
                for (int j1 = 0; j1 < N1; ++j1) v[j1] = col[N2 * j1 * W];
                rdft_plan<N1, true, N2>(v, twn);
#pragma unroll
                for (int k1 = 0; k1 < N1; ++k1) col[N2 * k1 * W] = (k1 && j2) ? twiddle<true>(v[k1], twn[j2 * k1]) : v[k1];
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < IT; ++i) {
                const int t = threadIdx.x + i * TB, w = t % W, k1 = t / W;
                if (t < N1 * W) {
#pragma unroll
                    for (int rr = 0; rr < NR; ++rr) {
                        const float2 *col = pbuf + (rr * D + N2 * k1) * W + w;
                        float2 u[N2];
#pragma unroll
                        for (int j2 = 0; j2 < N2; ++j2) u[j2] = col[j2 * W];
                        rdft_plan<N2, true, N1>(u, twn);
                        if (j0 + w < dH && (NR == 1 || b + rr < b1))
#pragma unroll
                            for (int k2 = 0; k2 < N2; ++k2)
                                dst[((size_t)rr * a.ngrp * D + k1 + N1 * k2) * dH + w] = u[k2];
                    }
                }
            }
            continue;
        }
        // inverse step 1: items (rotation, j2, w) -> U rows x = j2 + N2 j1
        for (int t = threadIdx.x; t < NR * N2 * W; t += TB) {
            const int w = t % W, rj = t / W, j2 = rj % N2, rr = rj / N2;
            const float2 *col = pbuf + (rr * D + N1 * j2) * W + w;
            float2 v[N1];
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) v[k1] = col[k1 * W];
            rdft<N1, true>(v);
            if (j0 + w < dH && (NR == 1 || b + rr < b1))
#pragma unroll
                for (int j1 = 0; j1 < N1; ++j1)
                    dst[((size_t)rr * a.ngrp * D + j2 + N2 * j1) * dH + w] = v[j1];
        }
    }
}

template <int NCH, int N1, int N2, bool PFA>
__global__ void __launch_bounds__(tb_shape<NCH, N1, N2, PFA>().threads, tb_shape<NCH, N1, N2, PFA>().ctas)
    k_tpass_b(const PassB2 a, int nb, int rper) {
    tpass_b<NCH, NCH, N1, N2, PFA>(a, 0, 0, nb, rper);
}
template <int N1, int N2, bool PFA>
__global__ void __launch_bounds__(tb_shape<4, N1, N2, PFA>().threads, tb_shape<4, N1, N2, PFA>().ctas)
    k_tpass_b_prob(const PassB2 a, int nb, int rper) {
    if (blockIdx.z == 0)
        tpass_b<3, 4, N1, N2, PFA>(a, 0, 0, nb, rper);
    else
        tpass_b<4, 4, N1, N2, PFA>(a, 3, 1, nb, rper);
}

// ---- pass C -------------------------------------------------------------------
template <int N1, int N2> __host__ __device__ constexpr int tc_warps() { return N1 * N2 <= 32 ? 2 : N1 * N2 <= 48 ? 4 : 8; }
template <int NGRP, int N1, int N2, bool PFA>
__host__ __device__ constexpr size_t smem_tc() {
    using G = TGeom<N1, N2, !PFA>;
    return (size_t)((G::D + 1) / 2 * 2) * sizeof(float2) + (size_t)NGRP * G::CS * sizeof(float2) +
           3 * 8 * sizeof(unsigned long long);
}

template <int NGRP, int SC, int N1, int N2, bool PFA>
__global__ void __launch_bounds__(tc_warps<N1, N2>() * 32) k_tpass_c(const PassC2 a) {
    using G = TGeom<N1, N2, !PFA>;
    constexpr int D = G::D, H = G::H, NP = G::NP, RS = G::RS, LS = G::LS, CS = G::CS, P2 = G::P2;
    constexpr int NW = tc_warps<N1, N2>(), PL = (NP + NW - 1) / NW;
    extern __shared__ __align__(16) unsigned char smem[];
    const int x = blockIdx.x, b = blockIdx.y, r = a.r0 + b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2 *twn = (float2 *)smem;
    float2 *buf = twn + (D + 1) / 2 * 2;   // [NGRP][2 NP][RS]
    unsigned long long *red = (unsigned long long *)(buf + NGRP * CS);
    twiddles_n(D, twn);
    __syncthreads();
    const float2 *src0 = a.U + ((size_t)b * NGRP * D + x) * (size_t)(D * H);
    if constexpr (!PFA) {
        // inverse y in the forward's order.  Step 1 from U: items (g, j2, kz) -> rows
        // N2 k1 + j2; step 2, in place: items (g, k1, kz), row y = k1 + N1 k2 stays at
        // N2 k1 + k2
        for (int t = threadIdx.x; t < NGRP * N2 * H; t += NW * 32) {
            const int kz = t % H, gj = t / H, j2 = gj % N2, g = gj / N2;
            const float2 *src = src0 + (size_t)g * (D * D * H) + j2 * H + kz;
            float2 v[N1];
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) v[j1] = src[N2 * j1 * H];
            rdft_plan<N1, true, N2>(v, twn);
            float2 *col = buf + g * CS + j2 * RS + kz;
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) col[N2 * k1 * RS] = (k1 && j2) ? twiddle<true>(v[k1], twn[j2 * k1]) : v[k1];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < NGRP * N1 * H; t += NW * 32) {
            int kz, gk;
            column_item<H>(t, NGRP * N1, kz, gk);
            const int k1 = gk % N1, g = gk / N1;
            float2 *col = buf + g * CS + N2 * k1 * RS + kz;
            float2 u[N2];
#pragma unroll
            for (int j2 = 0; j2 < N2; ++j2) u[j2] = col[j2 * RS];
            rdft_plan<N2, true, N1>(u, twn);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) col[k2 * RS] = u[k2];
        }
        __syncthreads();
    } else {
        // inverse y step 2 from U: items (g, k1, kz) -> rows N2 k1 + j2
        for (int t = threadIdx.x; t < NGRP * N1 * H; t += NW * 32) {
            const int kz = t % H, gk = t / H, k1 = gk % N1, g = gk / N1;
            const float2 *src = src0 + (size_t)g * (D * D * H) + k1 * H + kz;
            float2 u[N2];
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) u[k2] = src[N1 * k2 * H];
            rdft<N2, true>(u);
            float2 *col = buf + g * CS + N2 * k1 * RS + kz;
#pragma unroll
            for (int j2 = 0; j2 < N2; ++j2) col[j2 * RS] = (k1 && j2) ? cmulc(u[j2], twn[j2 * k1]) : u[j2];
        }
        __syncthreads();
        // inverse y step 1, in place: items (g, j2, kz) -> rows y = j2 + N2 j1
        for (int t = threadIdx.x; t < NGRP * N2 * H; t += NW * 32) {
            int kz, gj;
            column_item<H>(t, NGRP * N2, kz, gj);
            const int j2 = gj % N2, g = gj / N2;
            float2 *col = buf + g * CS + j2 * RS + kz;
            float2 v[N1];
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) v[k1] = col[N2 * k1 * RS];
            rdft<N1, true>(v);
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) col[N2 * j1 * RS] = v[j1];
        }
        __syncthreads();
    }
    const int p0 = warp * PL, pn = min(PL, NP - p0);   // pn <= 0: no line left for this warp
    unsigned long long best[3] = {0ull, 0ull, 0ull};
    // Best of one item's voxels, which come in ascending index order: the first of the
    // greatest scores, as offsets from the item's first voxel (half the instructions of
    // a 64-bit key per voxel); merged as keys once per item.
    // float_order as a signed value: the sum makes -0 a +0.
    int top[SC] = {}, at[SC] = {};
    auto take = [&](int s, float v, int off) {
        const int i = __float_as_int(__fadd_rn(v, 0.f)), o = i ^ (i >> 31 & 0x7fffffff);
        if (o > top[s]) {
            top[s] = o;
            at[s] = off;
        }
    };
    auto score = [&](float s0, float s1, int off) {
        take(0, s0, off);
        if (SC >= 2) take(SC >= 2 ? 1 : 0, s1, off);
        if (SC == 3) {
            const float sv = __fdiv_rn(__fsub_rn(s0, a.mix.vave), a.mix.vstd);
            const float sp = __fdiv_rn(__fsub_rn(s1, a.mix.pave), a.mix.pstd);
            take(SC == 3 ? 2 : 0, __fadd_rn(__fmul_rn(a.mix.one_minus_alpha, sv), __fmul_rn(a.mix.alpha, sp)), off);
        }
    };
    auto begin = [&]() {
#pragma unroll
        for (int s = 0; s < SC; ++s) top[s] = (int)0x80000000, at[s] = 0;
    };
    auto merge = [&](int y, int z) {
#pragma unroll
        for (int s = 0; s < SC; ++s)
            best[s] = max(best[s], (unsigned long long)((uint32_t)top[s] ^ 0x80000000u) << 32 |
                                       (0xffffffffu - (uint32_t)((x * D + y) * D + z + at[s])));
    };
    if constexpr (!PFA) {
        // z in the forward's order, each line in its own two rows' storage (elements
        // of k1 < KH in the first row's, the others in the second's): rows (2p, 2p + 1)
        // as one full line (Hermitian completion, DC and Nyquist imaginary parts
        // dropped); step 1: items (g, line, j2), whole lines per round, read before
        // they are written; step 2 and scores: items (line, k1) over every group
        constexpr int KH = (N1 + 1) / 2, LPR = 32 / N2;
        auto row_at = [](int y) { return (N2 * (y % N1) + y / N1) * RS; };
        const int lj2 = lane % N2, lq = lane / N2;
#pragma unroll 1
        for (int l0 = 0; l0 < NGRP * pn; l0 += LPR) {
            const int l = l0 + lq, g = NGRP == 2 ? l / max(pn, 1) : 0, p = p0 + l - g * pn;
            const bool on = lq < LPR && l < NGRP * pn;
            const bool hb = 2 * p + 1 < D;
            float2 *ra = buf + g * CS + row_at(2 * p), *rb = hb ? buf + g * CS + row_at(2 * p + 1) : buf + g * CS + D * RS;
            float2 v[N1];
            if (on) {
#pragma unroll
                for (int j1 = 0; j1 < N1; ++j1) {
                    const int k = lj2 + N2 * j1;
                    const bool low = k < H;
                    const int kk = low ? k : D - k;
                    float2 A = ra[kk], B = hb ? rb[kk] : make_float2(0.f, 0.f);
                    if (k == 0 || 2 * k == D) { A.y = 0.f; B.y = 0.f; }
                    v[j1] = low ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, B.x - A.y);
                }
                rdft_plan<N1, true, N2>(v, twn);
            }
            __syncwarp();
            if (on)
#pragma unroll
                for (int k1 = 0; k1 < N1; ++k1)
                    (k1 < KH ? ra + P2 * k1 : rb + P2 * (k1 - KH))[lj2] = (k1 && lj2) ? twiddle<true>(v[k1], twn[lj2 * k1]) : v[k1];
        }
        __syncwarp();
        for (int t = lane; t < pn * N1; t += 32) {
            const int k1 = t % N1, p = p0 + t / N1;
            const bool hb = 2 * p + 1 < D;
            const int at = k1 < KH ? row_at(2 * p) + P2 * k1 : (hb ? row_at(2 * p + 1) : D * RS) + P2 * (k1 - KH);
            float2 u0[N2], u1[N2];
#pragma unroll
            for (int j2 = 0; j2 < N2; ++j2) u0[j2] = buf[at + j2];
            rdft_plan<N2, true, N1>(u0, twn);
            if (NGRP == 2) {
#pragma unroll
                for (int j2 = 0; j2 < N2; ++j2) u1[j2] = buf[CS + at + j2];
                rdft_plan<N2, true, N1>(u1, twn);
            }
            begin();
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) score(u0[k2].x, NGRP == 2 ? u1[k2].x : 0.f, N1 * k2);
            if (hb)
#pragma unroll
                for (int k2 = 0; k2 < N2; ++k2) score(u0[k2].y, NGRP == 2 ? u1[k2].y : 0.f, D + N1 * k2);
            merge(2 * p, k1);
        }
    } else {
        // z: rows (2p, 2p + 1) as one full line (Hermitian completion, DC and Nyquist
        // imaginary parts dropped), inverse step 2 in the rows' own storage: items
        // (g, line, k1), whole lines per round, read before they are written
        constexpr int LPR = 32 / N1;
        constexpr bool LF = LPR % 4 == 0;   // line fastest: 4 lines fall in different banks
        const int lk1 = LF ? lane / LPR : lane % N1, lq = LF ? lane % LPR : lane / N1;
#pragma unroll 1
        for (int l0 = 0; l0 < NGRP * pn; l0 += LPR) {
            const int l = l0 + lq, g = NGRP == 2 ? l / max(pn, 1) : 0, p = p0 + l - g * pn;
            const bool on = lq < LPR && lk1 < N1 && l < NGRP * pn;
            float2 *line = buf + g * CS + p * LS;
            const bool hb = 2 * p + 1 < D;
            float2 u[N2];
            if (on) {
#pragma unroll
                for (int k2 = 0; k2 < N2; ++k2) {
                    const int k = lk1 + N1 * k2;
                    if (k < H) {
                        float2 A = line[k], B = hb ? line[RS + k] : make_float2(0.f, 0.f);
                        if (k == 0 || 2 * k == D) { A.y = 0.f; B.y = 0.f; }
                        u[k2] = make_float2(A.x - B.y, A.y + B.x);
                    } else {
                        const float2 A = line[D - k], B = hb ? line[RS + D - k] : make_float2(0.f, 0.f);
                        u[k2] = make_float2(A.x + B.y, B.x - A.y);
                    }
                }
                rdft<N2, true>(u);
            }
            __syncwarp();
            if (on)
#pragma unroll
                for (int j2 = 0; j2 < N2; ++j2)
                    line[P2 * lk1 + j2] = (lk1 && j2) ? cmulc(u[j2], twn[j2 * lk1]) : u[j2];
        }
        __syncwarp();
        // inverse z step 1 and scores: items (line, j2) over every group
        for (int t = lane; t < pn * N2; t += 32) {
            const int j2 = t / pn, p = p0 + t - j2 * pn;
            float2 v0[N1], v1[N1];
            const float2 *l0 = buf + p * LS + j2;
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) v0[k1] = l0[P2 * k1];
            rdft<N1, true>(v0);
            if (NGRP == 2) {
#pragma unroll
                for (int k1 = 0; k1 < N1; ++k1) v1[k1] = l0[CS + P2 * k1];
                rdft<N1, true>(v1);
            }
            begin();
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) score(v0[j1].x, NGRP == 2 ? v1[j1].x : 0.f, N2 * j1);
            if (2 * p + 1 < D)
#pragma unroll
                for (int j1 = 0; j1 < N1; ++j1) score(v0[j1].y, NGRP == 2 ? v1[j1].y : 0.f, D + N2 * j1);
            merge(2 * p, j2);
        }
    }
#pragma unroll
    for (int s = 0; s < SC; ++s) {
        const unsigned long long v = warp_max_u64(best[s]);
        if (lane == 0) red[s * 8 + warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < SC) {
        unsigned long long v = 0ull;
        for (int w = 0; w < NW; ++w) v = max(v, red[threadIdx.x * 8 + w]);
        atomicMax(&a.keys[(size_t)r * a.nscore + threadIdx.x], v);
    }
}

}  // namespace vg
