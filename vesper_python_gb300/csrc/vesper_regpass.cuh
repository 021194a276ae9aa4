// Search passes with register-resident line FFTs, for the grid sides compiled
// in (vesper_sides_*.cu; every other side uses the radix-stage passes of
// vesper_passes.cuh): whole lines in registers for sides up to 32 (here), two
// register steps per line above (vesper_tilepass.cuh).  Same inputs, outputs
// and layouts as the radix-stage passes.
#pragma once

#include "vesper_regfft.cuh"
#include "vesper_tilegather.cuh"
#include "vesper_tilepass.cuh"

namespace vg {

// ---------------------------------------------------------------------------
// Pass A for sides up to 32 with whole lines in registers, a few x planes per CTA:
// the gather, then one packed z line per thread (DFT + unpack in registers),
// then one y column per thread (DFT in registers, straight to S).
// Several channels: one plane on 64 threads (measured at side 30, 3 channels: 0.157 us
// per rotation, 0.182 with 2 planes on 96 threads, although those leave fewer idle;
// side 32 0.199 and 0.265 with 5 planes).  One channel has 16 lines a plane, so there
// the fewest idle threads over both phases and the last CTA's planes decide, up to 128
// threads (side 30: 0.135 -> 0.125 us).
struct LineShape {
    int planes, threads;
};
template <int SRC, int D>
__host__ __device__ constexpr LineShape line_a_shape() {
    constexpr int C = src_nch<SRC>(), NP = (D + 1) / 2, H = D / 2 + 1;
    LineShape best{1, 64};
    if (C > 1) return best;
    long long bn = 0, bd = 1;   // used over held thread slots
    for (int p = 1; p <= 6; ++p)
        for (int t = 64; t <= 128; t += 32) {
            const long long used = (long long)D * C * (NP + H);
            const long long held = (long long)((D + p - 1) / p) * t * ((p * C * NP + t - 1) / t + (p * C * H + t - 1) / t);
            if (used * bd > bn * held) {
                bn = used;
                bd = held;
                best = LineShape{p, t};
            }
        }
    return best;
}

template <int D>
struct LineGeom {
    static constexpr int H = D / 2 + 1, NP = (D + 1) / 2, Hp = H | 1;
    static constexpr int LS = 2 * Hp + 1;   // packed-line stride (odd)
    static constexpr int PS = NP * LS;      // plane stride per channel
};
template <int SRC, int D>
__host__ __device__ constexpr size_t smem_ra_line() {
    return ((size_t)line_a_shape<SRC, D>().planes * src_nch<SRC>() * LineGeom<D>::PS + D) * sizeof(float2);
}

// T: the block's threads (prob mode's two kinds of channels share a launch).
template <int SRC, int D, bool PFA, int PL, int T>
__device__ __forceinline__ void rpass_a_line(const PassA2 &a, int c0) {
    using L = LineGeom<D>;
    constexpr int H = L::H, NP = L::NP, Hp = L::Hp, LS = L::LS, PS = L::PS, NCH = src_nch<SRC>();
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *buf = (float2 *)smem;   // [PL][NCH][NP][LS]
    float2 *twn = buf + PL * NCH * PS;
    const int x0 = blockIdx.x * PL, b = blockIdx.y, r = a.r0 + b, pn = min(PL, D - x0);
    if constexpr (!PFA) twiddles_n(D, twn);
    if (x0 == 0 && c0 == 0 && threadIdx.x < a.nscore) a.keys[(size_t)r * a.nscore + threadIdx.x] = 0ull;
    float F[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) F[i] = __ldg(a.rotmats + (size_t)r * 9 + i);
    gather_planes<SRC, D, LS, PS, T / 32, false>(a, F, b, x0, pn, buf, [](int z) { return z; });
    __syncthreads();
    // z: one packed line per thread; DFT and unpack into rows 2p (offset 0)
    // and 2p + 1 (offset Hp) of the line's own storage
    for (int t = threadIdx.x; t < pn * NCH * NP; t += T) {
        const int p = t % NP, c = t / NP;   // c: plane and channel
        float2 *line = buf + c * PS + p * LS;
        float2 v[D];
#pragma unroll
        for (int j = 0; j < D; ++j) v[j] = line[j];
        line_dft<D, D, false, PFA, true>(v, twn);   // largest prime power first (faster here)
        const bool two = 2 * p + 1 < D;
#pragma unroll
        for (int k = 0; k < H; ++k) {
            float2 A, B;
            unpack_pair(v[k], v[(D - k) % D], A, B);
            line[k] = A;
            line[Hp + k] = two ? B : make_float2(0.f, 0.f);
        }
    }
    __syncthreads();
    // y: one column (plane, channel, kz) per thread -> S rows ky
    for (int t = threadIdx.x; t < pn * NCH * H; t += T) {
        const int kz = t % H, pc = t / H, pl = pc / NCH, c = pc - pl * NCH;
        const float2 *pln = buf + pc * PS + kz;
        float2 v[D];
#pragma unroll
        for (int y = 0; y < D; ++y) v[y] = pln[(y >> 1) * LS + (y & 1) * Hp];
        line_dft<D, D, false, PFA, true>(v, twn);   // largest prime power first (faster here)
        float2 *dst = a.S + (((size_t)b * a.nch + c0 + c) * D + x0 + pl) * (size_t)D * H + kz;
#pragma unroll
        for (int ky = 0; ky < D; ++ky) dst[(size_t)ky * H] = v[ky];
    }
}

// At most 128 registers a thread (8 CTAs of 64 threads per SM).
template <int SRC, int D, bool PFA>
__global__ void __launch_bounds__(line_a_shape<SRC, D>().threads, 512 / line_a_shape<SRC, D>().threads)
    k_rpass_a_line(const PassA2 a) {
    constexpr LineShape s = line_a_shape<SRC, D>();
    rpass_a_line<SRC, D, PFA, s.planes, s.threads>(a, 0);
}
// prob mode: the vector channels and the probability channels in CTAs of their own
template <int D, bool PFA>
__global__ void __launch_bounds__(64, 8) k_rpass_a_line_prob(const PassA2 a) {
    if (blockIdx.z == 0)
        rpass_a_line<kSrcVec, D, PFA, 1, 64>(a, 0);
    else
        rpass_a_line<kSrcProb, D, PFA, 1, 64>(a, 3);
}

// A whole line's DFT in registers with the arithmetic of the two register steps
// (vesper_tilepass.cuh, PFA): N1 points, twiddles, N2 points, or the inverse's
// opposite order.  For the passes whose sides up to 32 were two-step kernels.
template <int N1, int N2, bool INV>
__device__ __forceinline__ void line_dft_two(float2 *v, const float2 *twn) {
    constexpr int D = N1 * N2;
    float2 w[D];   // [j2][k1]
    if constexpr (!INV) {
#pragma unroll
        for (int j2 = 0; j2 < N2; ++j2) {
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) w[N1 * j2 + j1] = v[j2 + N2 * j1];
            rdft<N1, false>(w + N1 * j2);
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1)
                if (k1 && j2) w[N1 * j2 + k1] = cmul(w[N1 * j2 + k1], twn[j2 * k1]);
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
        float2 u[N2];
#pragma unroll
        for (int i = 0; i < N2; ++i) u[i] = INV ? v[k1 + N1 * i] : w[N1 * i + k1];
        rdft<N2, INV>(u);
#pragma unroll
        for (int i = 0; i < N2; ++i) {
            if constexpr (INV)
                w[N1 * i + k1] = (k1 && i) ? cmulc(u[i], twn[i * k1]) : u[i];
            else
                v[k1 + N1 * i] = u[i];
        }
    }
    if constexpr (INV) {
#pragma unroll
        for (int j2 = 0; j2 < N2; ++j2) {
            rdft<N1, true>(w + N1 * j2);
#pragma unroll
            for (int j1 = 0; j1 < N1; ++j1) v[j2 + N2 * j1] = w[N1 * j2 + j1];
        }
    }
}
template <int N1, int N2, bool INV, bool PFA, bool TWO>
__device__ __forceinline__ void line_dft_as(float2 *v, const float2 *twn) {
    if constexpr (TWO)
        line_dft_two<N1, N2, INV>(v, twn);
    else
        line_dft<N1 * N2, N1 * N2, INV, PFA>(v, twn);
}

// ---------------------------------------------------------------------------
// Pass B for sides up to 32: one spectrum column j =
// ky H + kz per thread, whole x lines in registers -- for every channel the
// forward x DFT of its S column, times conj(T) added into the column's sum,
// then the inverse x DFT of the sum straight to U.  No shared memory.
constexpr int kLineBThreads = 64;  // fewer idle threads in the last CTA of each rotation (measured: 64 beat 128, 256)

template <int NCH, int N1, int N2, bool PFA, bool TWO>
__device__ __forceinline__ void rpass_b_line(const PassB2 &a, int c0, int grp) {
    constexpr int D = N1 * N2, H = D / 2 + 1, dH = D * H;
    __shared__ float2 twn[PFA && !TWO ? 1 : D];
    if constexpr (!PFA || TWO) {
        twiddles_n(D, twn);
        __syncthreads();
    }
    const int j = blockIdx.x * kLineBThreads + threadIdx.x, b = blockIdx.y;
    if (j >= dH) return;
    const float2 *src = a.S + ((size_t)b * a.nch + c0) * D * dH + j;
    float2 acc[D];
#pragma unroll
    for (int k = 0; k < D; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int c = 0; c < NCH; ++c) {
        float2 v[D];
#pragma unroll
        for (int x = 0; x < D; ++x) v[x] = src[(size_t)(c * D + x) * dH];
        line_dft_as<N1, N2, false, PFA, TWO>(v, twn);
        const float2 *T = a.T + (size_t)(c0 + c) * D * dH + j;
#pragma unroll
        for (int k = 0; k < D; ++k) acc[k] = cadd(acc[k], cmul(T[(size_t)k * dH], v[k]));
    }
    line_dft_as<N1, N2, true, PFA, TWO>(acc, twn);
    float2 *dst = a.U + ((size_t)b * a.ngrp + grp) * D * dH + j;
#pragma unroll
    for (int x = 0; x < D; ++x) dst[(size_t)x * dH] = acc[x];
}

template <int NCH, int N1, int N2, bool PFA>
__global__ void __launch_bounds__(kLineBThreads) k_rpass_b_line(const PassB2 a) {
    rpass_b_line<NCH, N1, N2, PFA, false>(a, 0, 0);
}
template <int N1, int N2, bool PFA>
__global__ void __launch_bounds__(kLineBThreads) k_rpass_b_line_prob(const PassB2 a) {
    if (blockIdx.z == 0)
        rpass_b_line<3, N1, N2, PFA, PFA>(a, 0, 0);
    else
        rpass_b_line<4, N1, N2, PFA, PFA>(a, 3, 1);
}

// ---------------------------------------------------------------------------
// Pass C for sides up to 32 with one score group and one score: several
// x-planes per CTA, whole lines in registers.  Phase y: one (plane, kz) column
// per thread, its D values read from U, inverse DFT, rows y to shared memory;
// phase z: one (plane, row pair) per thread, the two rows' half spectra packed
// into one complex line (Hermitian completion, DC and Nyquist imaginary parts
// dropped), inverse DFT (real part row 2p, imaginary part row 2p + 1), the
// scores' first-index argmax keys; one barrier between the phases.  With
// several planes per CTA both phases keep most threads busy.
// Row pairs sit 2 H + 1 elements apart: lanes of the z phase run over row pairs, and
// with a stride of 2 H, 32 at side 30, all of them fell in one bank.
// Planes: the divisor of D with the fewest idle threads over both phases (a column
// per thread, rounded up to whole warps, at most 128).  Microseconds per rotation,
// mode V: side 30 0.065 (2 planes; 0.092 for the two-step kernel with block
// barriers between its steps), side 28 0.057 (4), side 32 0.080 (4; 0.104 with 7
// planes on 128 threads, although those leave fewer idle).
template <int D> __host__ __device__ constexpr bool line_c_used() { return D <= kLineSide; }
template <int D> __host__ __device__ constexpr LineShape line_c_shape() {
    constexpr int NP = (D + 1) / 2, H = D / 2 + 1;
    LineShape best{1, 32};
    for (int p = 1; p <= D; ++p) {
        const int t = (p * H + 31) / 32 * 32;
        if (D % p == 0 && t <= 128 && p * (NP + H) * best.threads > best.planes * (NP + H) * t) best = LineShape{p, t};
    }
    return best;
}
template <int D> __host__ __device__ constexpr int line_c_planes() { return line_c_shape<D>().planes; }
template <int D> __host__ __device__ constexpr int line_c_threads() { return line_c_shape<D>().threads; }

template <int D, int PL>
__host__ __device__ constexpr size_t smem_rc_line() {
    return ((size_t)PL * ((D + 1) / 2) * (2 * (D / 2 + 1) + 1) + D + 1) * sizeof(float2) + 2 * sizeof(unsigned long long);
}

template <int N1, int N2, bool PFA>
__global__ void __launch_bounds__(line_c_threads<N1 * N2>()) k_rpass_c_line(const PassC2 a) {
    constexpr int D = N1 * N2, H = D / 2 + 1, NP = (D + 1) / 2, PL = line_c_planes<D>(), LS = 2 * H + 1;
    constexpr bool TWO = PFA && D % 4 != 0;
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *rows = (float2 *)smem;   // [PL][NP][LS]
    unsigned long long *red = (unsigned long long *)(rows + (size_t)PL * NP * LS);   // [2]
    const int x0 = blockIdx.x * PL, b = blockIdx.y, r = a.r0 + b;
    float2 *twn = (float2 *)(red + 2);
    if constexpr (!PFA || TWO) {
        twiddles_n(D, twn);
        __syncthreads();
    }
    if (threadIdx.x < 2) red[threadIdx.x] = 0ull;
    // y: inverse DFT of every (plane, kz) column
    for (int t = threadIdx.x; t < PL * H; t += blockDim.x) {
        const int pl = t / H, kz = t - pl * H, x = x0 + pl;
        if (x >= D) continue;
        const float2 *src = a.U + ((size_t)b * D + x) * (size_t)D * H + kz;
        float2 v[D];
#pragma unroll
        for (int ky = 0; ky < D; ++ky) v[ky] = src[(size_t)ky * H];
        line_dft_as<N1, N2, true, PFA, TWO>(v, twn);
        float2 *dst = rows + (size_t)pl * NP * LS + kz;
#pragma unroll
        for (int y = 0; y < D; ++y) dst[(y >> 1) * LS + (y & 1) * H] = v[y];
    }
    __syncthreads();
    // z: row pairs (2p, 2p + 1), inverse complex DFT, scores
    unsigned long long best = 0ull;
    for (int t = threadIdx.x; t < PL * NP; t += blockDim.x) {
        const int pl = t / NP, p = t - pl * NP, x = x0 + pl, y = 2 * p;
        if (x >= D) continue;
        const float2 *r0 = rows + (pl * NP + p) * LS;
        const bool hb = y + 1 < D;
        const float2 *r1 = r0 + H;
        float2 u[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            if (k < H) {
                float2 A = r0[k], B = hb ? r1[k] : make_float2(0.f, 0.f);
                if (k == 0 || 2 * k == D) { A.y = 0.f; B.y = 0.f; }
                u[k] = make_float2(A.x - B.y, A.y + B.x);
            } else {
                const float2 A = r0[D - k], B = hb ? r1[D - k] : make_float2(0.f, 0.f);
                u[k] = make_float2(A.x + B.y, B.x - A.y);
            }
        }
        line_dft_as<N1, N2, true, PFA, TWO>(u, twn);
        const uint32_t base = (uint32_t)((x * D + y) * D);
#pragma unroll
        for (int z = 0; z < D; ++z) {
            best = max(best, make_key(u[z].x, base + z));
            if (hb) best = max(best, make_key(u[z].y, base + D + z));
        }
    }
    best = warp_max_u64(best);
    if ((threadIdx.x & 31) == 0) atomicMax(&red[0], best);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&a.keys[(size_t)r * a.nscore], red[0]);
}

// ---- one compiled side of the register passes, as vesper_search.cu calls it ----
// Kinds: 0 vectors, 1 values (modes O, C, P), 2 an already rotated field (mode L),
// 3 vectors and probabilities.
struct RegEntry {
    int d, kinds;   // kinds: a bit for each that the entry has
    void (*a[4])(int nb, cudaStream_t, const PassA2 &);   // nb rotations
    void (*b[4])(int nb, cudaStream_t, const PassB2 &);
    void (*c[4])(int nb, cudaStream_t, const PassC2 &);
};
constexpr int kVec = 1, kVal = 2, kPlain = 4, kProb = 8;
__host__ inline int reg_kind(int mode) {
    return mode == VESPER_MODE_VEC ? 0 : mode == VESPER_MODE_PROB ? 3 : mode == VESPER_MODE_LAPLACIAN ? 2 : 1;
}

// Rotations that one CTA of pass B takes one after another: as many as leave
// two full waves of CTAs (its target values are read once for all of them).
inline int tb_rotations(int nbx, int nb) {
    const long long ctas = (long long)nbx * nb;
    return (int)std::max(1LL, std::min(8LL, ctas / (2 * 152 * 4)));
}

// PFA: line DFTs with coprime factors split without twiddles.  Else they repeat
// the radix-stage passes' arithmetic, which these sides and modes ran before, bit
// for bit (a search's best translation, and Overlap's exact ties above all, hang
// on the rounding of the scores); N2 is then the plan's last radix.
template <int N1, int N2, bool PFA, int KINDS>
struct RegSide {
    static constexpr int D = N1 * N2, H = D / 2 + 1;
    static constexpr bool kLine = D <= kLineSide;
    static_assert(PFA || kLine || plan_last<D>() == N2, "the second step is the plan's last stage");

    template <int SRC>
    static void a(int nb, cudaStream_t st, const PassA2 &p) {
        if constexpr (kLine) {
            constexpr size_t sm = smem_ra_line<SRC, D>();
            allow_smem(k_rpass_a_line<SRC, D, PFA>, sm);
            constexpr LineShape sh = line_a_shape<SRC, D>();
            k_rpass_a_line<SRC, D, PFA><<<dim3((D + sh.planes - 1) / sh.planes, nb), sh.threads, sm, st>>>(p);
        } else {
            constexpr size_t sm = smem_ta<SRC, N1, N2>();
            allow_smem(k_tpass_a<SRC, N1, N2, PFA>, sm);
            k_tpass_a<SRC, N1, N2, PFA><<<dim3(D, nb), ta_warps<N1, N2>() * 32, sm, st>>>(p);
        }
    }
    static void a_prob(int nb, cudaStream_t st, const PassA2 &p) {
        if constexpr (kLine) {
            constexpr size_t sm = (4 * LineGeom<D>::PS + D) * sizeof(float2);
            allow_smem(k_rpass_a_line_prob<D, PFA>, sm);
            k_rpass_a_line_prob<D, PFA><<<dim3(D, nb, 2), 64, sm, st>>>(p);
        } else {
            constexpr size_t sm = smem_ta<kSrcProb, N1, N2>();
            allow_smem(k_tpass_a_prob<N1, N2, PFA>, sm);
            k_tpass_a_prob<N1, N2, PFA><<<dim3(D, nb, 2), ta_warps<N1, N2>() * 32, sm, st>>>(p);
        }
    }
    template <int NCH>
    static void b(int nb, cudaStream_t st, const PassB2 &p) {
        if constexpr (kLine) {
            k_rpass_b_line<NCH, N1, N2, PFA>
                <<<dim3((D * H + kLineBThreads - 1) / kLineBThreads, nb), kLineBThreads, 0, st>>>(p);
        } else {
            constexpr BShape s = tb_shape<NCH, N1, N2, PFA>();
            constexpr int nbx = (D * H + s.cols - 1) / s.cols;
            constexpr size_t sm = smem_tb<NCH, N1, N2, PFA>();
            const int rper = s.side * tb_rotations(nbx, nb / s.side);
            allow_smem(k_tpass_b<NCH, N1, N2, PFA>, sm);
            k_tpass_b<NCH, N1, N2, PFA><<<dim3(nbx, (nb + rper - 1) / rper), s.threads, sm, st>>>(p, nb, rper);
        }
    }
    static void b_prob(int nb, cudaStream_t st, const PassB2 &p) {
        if constexpr (kLine) {
            k_rpass_b_line_prob<N1, N2, PFA>
                <<<dim3((D * H + kLineBThreads - 1) / kLineBThreads, nb, 2), kLineBThreads, 0, st>>>(p);
        } else {
            constexpr BShape s = tb_shape<4, N1, N2, PFA>();
            constexpr int nbx = (D * H + s.cols - 1) / s.cols;
            constexpr size_t sm = smem_tb<4, N1, N2, PFA>();
            const int rper = s.side * tb_rotations(2 * nbx, nb / s.side);
            allow_smem(k_tpass_b_prob<N1, N2, PFA>, sm);
            k_tpass_b_prob<N1, N2, PFA>
                <<<dim3(nbx, (nb + rper - 1) / rper, 2), s.threads, sm, st>>>(p, nb, rper);
        }
    }
    template <int NGRP, int SC>
    static void tc(int nb, cudaStream_t st, const PassC2 &p) {
        constexpr size_t sm = smem_tc<NGRP, N1, N2, PFA>();
        allow_smem(k_tpass_c<NGRP, SC, N1, N2, PFA>, sm);
        k_tpass_c<NGRP, SC, N1, N2, PFA><<<dim3(D, nb), tc_warps<N1, N2>() * 32, sm, st>>>(p);
    }
    static void c(int nb, cudaStream_t st, const PassC2 &p) {
        if constexpr (line_c_used<D>()) {
            constexpr int PL = line_c_planes<D>();
            constexpr size_t sm = smem_rc_line<D, PL>();
            allow_smem(k_rpass_c_line<N1, N2, PFA>, sm);
            k_rpass_c_line<N1, N2, PFA><<<dim3((D + PL - 1) / PL, nb), line_c_threads<D>(), sm, st>>>(p);
        } else {
            tc<1, 1>(nb, st, p);
        }
    }
    static void c_prob(int nb, cudaStream_t st, const PassC2 &p) {
        if (p.nscore == 2)
            tc<2, 2>(nb, st, p);
        else
            tc<2, 3>(nb, st, p);
    }
    static RegEntry entry() {
        RegEntry e{};
        e.d = D;
        e.kinds = KINDS;
        if constexpr ((KINDS & kVec) != 0) e.a[0] = &a<kSrcVec>, e.b[0] = &b<3>, e.c[0] = &c;
        if constexpr ((KINDS & kVal) != 0) e.a[1] = &a<kSrcVal>, e.b[1] = &b<1>, e.c[1] = &c;
        if constexpr ((KINDS & kPlain) != 0) e.a[2] = &a<kSrcPlain>, e.b[2] = &b<1>, e.c[2] = &c;
        if constexpr ((KINDS & kProb) != 0) e.a[3] = &a_prob, e.b[3] = &b_prob, e.c[3] = &c_prob;
        return e;
    }
};

// the tables of vesper_sides_*.cu: the entry of side d and kind, or null
const RegEntry *find_reg_pfa_a(int d, int kind);
const RegEntry *find_reg_pfa_b(int d, int kind);
const RegEntry *find_reg_a(int d, int kind);
const RegEntry *find_reg_b(int d, int kind);
const RegEntry *find_reg_c(int d, int kind);
const RegEntry *find_reg_d(int d, int kind);
const RegEntry *find_reg_e(int d, int kind);
const RegEntry *find_reg_f(int d, int kind);
const RegEntry *find_reg_g(int d, int kind);
const RegEntry *find_reg_h(int d, int kind);
const RegEntry *find_reg_i(int d, int kind);
const RegEntry *find_reg_j(int d, int kind);
const RegEntry *find_reg_k(int d, int kind);
const RegEntry *find_reg_l(int d, int kind);

inline const RegEntry *find_in(const RegEntry *table, int n, int d, int kind) {
    for (int i = 0; i < n; ++i)
        if (table[i].d == d && (table[i].kinds >> kind & 1)) return &table[i];
    return nullptr;
}

}  // namespace vg
