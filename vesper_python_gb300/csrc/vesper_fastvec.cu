// fastVEC on the GPU: the Gaussian-weighted density and unit vector of every
// destination voxel of the coarse grid (doFastVEC / calc,
// VESPER_1_prob_new.py:121-142, :180-257).
//
// The reference sums, for each destination voxel at source position pos,
//   v = src[p] * exp(-1.5 |p - pos|^2 fsiv)
// over the box [int(pos - fmaxd) v 0, int(pos + fmaxd + 1) ^ S) on each axis,
// together with v * p.  Both the weight and the box factor per axis, and pos
// on axis a depends only on the destination index on that axis, so the sums
// are three successive 1-D banded contractions (z, then y, then x):
//   A0[xp][yp][z] = sum_zp wz[z][zp] src[xp][yp][zp]      A1 = same with zp wz
//   B0[xp][y][z]  = sum_yp wy[y][yp] A0                    B1 = yp wy A0, B2 = wy A1
//   D = sum_xp wx B0, Px = sum xp wx B0, Py = sum wx B1, Pz = sum wx B2
// with w = exp(-1.5 r^2 fsiv) per axis (the product of the three per-axis
// factors is the reference's exp of the sum up to rounding).  The per-voxel
// skip tests (pos inside the source, src[int(pos)] != 0) and the
// normalisation follow the reference operation by operation.
//
// Cost: S0 S1 d WB + S0 d^2 WB + d^3 WB multiply-adds (x2..4) instead of
// d^3 WB^3 exponentials, WB = band width <= 2 fmaxd + 2.
//
// Arithmetic.  The reference sums in float64, which runs at 1/64 of the
// float32 rate on this part.  The contractions therefore carry every partial
// sum as an unevaluated pair of float32 values hi + lo ("double-single" or
// float-float numbers, Dekker 1971): products by TwoProd (the rounding error
// of hi * v recovered exactly with one fmaf), sums by Knuth's TwoSum followed by
// a FastTwoSum renormalisation after every term, about 2^-46 relative per
// operation.  Every term is non-negative (the thresholded source is >= 0;
// weights and positions are positive), so nothing cancels inside a sum.  The
// weights are computed in float64 and split into pairs; each voxel's finish
// (ratios, norm, unit vector) runs in float64 on the pair sums.  Against the
// float64 restatement of the reference loop this gives densities within 1e-13
// relative and the same float32 vectors.  A pair cannot hold a weight below
// the float32 normal range to full precision, so geometries whose smallest
// band weight exp(-1.5 (fmaxd + 1)^2 fsiv) is below 2^-70 (dreso / src_width
// below about 0.8) run the same contractions in float64 instead.
#include <algorithm>
#include <cmath>

#include "vesper_common.cuh"

namespace vg {

struct AxisTables {
    // per axis a and destination index i (d entries each)
    double *pos;     // [3][d]
    int *stp;        // [3][d]
    int *len;        // [3][d] endp - stp (>= 0)
    int *idx;        // [3][d] int(pos) if 0 <= pos < S else -1
    double *w;       // [3][WB][d]  weight of band entry k
    double *wp;      // [3][WB][d]  weight * (stp + k)
    float2 *wf;      // [3][WB][d]  w as a float-float pair (hi, lo)
    float2 *wpf;     // [3][WB][d]  wp as a pair
    // float-float stages, written by k_fvf_scan
    int *rlo, *rhi;          // [S0] first and last row of plane xp that holds a non-zero value (rhi -1: none)
    int *list;               // [S0 S1] the rows that do, any order
    unsigned char *rowf;     // [S0 S1] 1 where a row does
    unsigned char *need;     // [d d] 1 where column (y, z) has a voxel that passes the skip tests
    int *voxels;             // [d^3] those voxels, any order
    int *count;              // [4] rows listed, voxels listed, first and last plane with a row
};

struct FvGeom {
    int S[3];
    int d, WB;
    double sw, dw, fsiv, fmaxd;
    double sorig[3], dorig[3];
};

// Block (i, a): destination index i on axis a; its threads share the band
// entries k (the exponentials), each computing the same position and band.
__global__ void k_fv_tables(const FvGeom g, AxisTables t) {
    const int i = blockIdx.x;
    const int a = blockIdx.y;
    if (i >= g.d) return;
    if (a == 0)   // clear the lists: block i takes planes i*128 + tid + m*128*d
        for (int xp = i * blockDim.x + threadIdx.x; xp < g.S[0]; xp += g.d * blockDim.x) {
            t.rlo[xp] = g.S[1];
            t.rhi[xp] = -1;
        }
    if (a == 1)
        for (int z = threadIdx.x; z < g.d; z += blockDim.x) t.need[i * g.d + z] = 0;
    if (a == 2 && i == 0 && threadIdx.x < 4) t.count[threadIdx.x] = threadIdx.x == 2 ? g.S[0] : threadIdx.x == 3 ? -1 : 0;
    // (xyz_arr * dest_xwidth + dest_orig - src_orig) / src_xwidth
    double p = __dmul_rn((double)i, g.dw);
    p = __dadd_rn(p, g.dorig[a]);
    p = __dsub_rn(p, g.sorig[a]);
    p = __ddiv_rn(p, g.sw);
    const int o = a * g.d + i;
    int stp = __double2int_rz(__dsub_rn(p, g.fmaxd));
    if (stp < 0) stp = 0;
    int endp = __double2int_rz(__dadd_rn(__dadd_rn(p, g.fmaxd), 1.0));
    if (endp >= g.S[a]) endp = g.S[a];
    const int len = max(0, min(endp - stp, g.WB));
    if (threadIdx.x == 0) {
        t.pos[o] = p;
        t.idx[o] = (p >= 0.0 && p < (double)g.S[a]) ? (int)p : -1;
        t.stp[o] = stp;
        t.len[o] = len;
    }
    for (int k = threadIdx.x; k < g.WB; k += blockDim.x) {
        double w = 0.0;
        if (k < len) {
            double r = __dsub_rn((double)(stp + k), p);
            r = __dmul_rn(r, r);
            w = exp(__dmul_rn(__dmul_rn(-1.5, r), g.fsiv));
        }
        const size_t wo = ((size_t)a * g.WB + k) * g.d + i;
        const double wp = __dmul_rn(w, (double)(stp + k));
        t.w[wo] = w;
        t.wp[wo] = wp;
        // hi = w rounded to float32; lo = the (exact) remainder rounded to float32
        const float wh = __double2float_rn(w), wph = __double2float_rn(wp);
        t.wf[wo] = make_float2(wh, __double2float_rn(__dsub_rn(w, (double)wh)));
        t.wpf[wo] = make_float2(wph, __double2float_rn(__dsub_rn(wp, (double)wph)));
    }
}

// ---- float-float helpers (all operations explicitly rounded, so the compiler
// neither fuses nor reorders them) ------------------------------------------------
// (sh, sl) += (th, tl): TwoSum of the high parts, the low parts added to the
// error, then FastTwoSum to renormalise
__device__ __forceinline__ void ff_add(float &sh, float &sl, float th, float tl) {
    const float s = __fadd_rn(sh, th);
    const float bb = __fsub_rn(s, sh);
    float e = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bb)), __fsub_rn(th, bb));
    e = __fadd_rn(e, __fadd_rn(sl, tl));
    sh = __fadd_rn(s, e);
    sl = __fsub_rn(e, __fsub_rn(sh, s));
}

// (h, l) * v for a float32 v: TwoProd of h * v, plus l * v in the low part
__device__ __forceinline__ void ff_mul_f(float h, float l, float v, float &ph, float &pl) {
    ph = __fmul_rn(h, v);
    pl = __fmaf_rn(l, v, __fmaf_rn(h, v, -ph));
}

// (ah, al) * (bh, bl): TwoProd of the high parts plus both cross terms
__device__ __forceinline__ void ff_mul(float2 a, float2 b, float &ph, float &pl) {
    ph = __fmul_rn(a.x, b.x);
    float e = __fmaf_rn(a.x, b.x, -ph);
    e = __fmaf_rn(a.x, b.y, e);
    pl = __fmaf_rn(a.y, b.x, e);
}

// stage 1: contract z.  Block = RB source rows (xp, yp), all d outputs.
constexpr int kRB = 8;
__global__ void __launch_bounds__(256) k_fv_z(const float *src, const FvGeom g, const AxisTables t, double *A0,
                                              double *A1) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int S2 = g.S[2], d = g.d;
    const size_t nrows = (size_t)g.S[0] * g.S[1];
    const size_t row0 = (size_t)blockIdx.x * kRB;
    float *rows = (float *)smem;
    __shared__ int nz[kRB];   // row holds a non-zero value (thresholded maps are mostly empty rows)
    if (threadIdx.x < kRB) nz[threadIdx.x] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < kRB * S2; e += blockDim.x) {
        const size_t r = row0 + e / S2;
        const float v = r < nrows ? src[r * S2 + (e % S2)] : 0.f;
        rows[e] = v;
        if (v != 0.f) nz[e / S2] = 1;
    }
    __syncthreads();
    const int *stp = t.stp + 2 * d, *len = t.len + 2 * d;
    const double *w = t.w + (size_t)2 * g.WB * d, *wp = t.wp + (size_t)2 * g.WB * d;
    for (int o = threadIdx.x; o < kRB * d; o += blockDim.x) {
        const int rr = o / d, z = o - rr * d;
        const size_t r = row0 + rr;
        if (r >= nrows) continue;
        if (!nz[rr]) {   // an all-zero row: the sums are +0.0, as the loop would give
            A0[r * d + z] = 0.0;
            A1[r * d + z] = 0.0;
            continue;
        }
        const float *row = rows + rr * S2 + stp[z];
        const int n = len[z];
        double s0 = 0.0, s1 = 0.0;
        for (int k = 0; k < n; ++k) {
            const double v = (double)row[k];
            s0 = fma(v, w[(size_t)k * d + z], s0);
            s1 = fma(v, wp[(size_t)k * d + z], s1);
        }
        A0[r * d + z] = s0;
        A1[r * d + z] = s1;
    }
}

// stage 2: contract y.  Block = (xp, z tile of ZT).
constexpr int kZT = 32;
__global__ void __launch_bounds__(256) k_fv_y(const FvGeom g, const AxisTables t, const double *A0, const double *A1,
                                              double *B0, double *B1, double *B2) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int S1 = g.S[1], d = g.d;
    const int xp = blockIdx.y, z0 = blockIdx.x * kZT;
    const int zn = min(kZT, d - z0);
    double *a0 = (double *)smem;
    double *a1 = a0 + (size_t)S1 * kZT;
    __shared__ int any;   // the tile holds a non-zero partial sum (planes outside the map hold none)
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < S1 * kZT; e += blockDim.x) {
        const int yp = e / kZT, zz = e - yp * kZT;
        const size_t gi = ((size_t)xp * S1 + yp) * d + z0 + zz;
        const double v0 = zz < zn ? A0[gi] : 0.0, v1 = zz < zn ? A1[gi] : 0.0;
        a0[e] = v0;
        a1[e] = v1;
        if (v0 != 0.0 || v1 != 0.0) any = 1;
    }
    __syncthreads();
    if (!any) {   // every sum is +0.0, as the loop below would give (A0, A1 >= +0.0)
        for (int o = threadIdx.x; o < d * kZT; o += blockDim.x) {
            const int y = o / kZT, zz = o - y * kZT;
            if (zz >= zn) continue;
            const size_t go = ((size_t)xp * d + y) * d + z0 + zz;
            B0[go] = 0.0;
            B1[go] = 0.0;
            B2[go] = 0.0;
        }
        return;
    }
    const int *stp = t.stp + d, *len = t.len + d;
    const double *w = t.w + (size_t)g.WB * d, *wp = t.wp + (size_t)g.WB * d;
    for (int o = threadIdx.x; o < d * kZT; o += blockDim.x) {
        const int y = o / kZT, zz = o - y * kZT;
        if (zz >= zn) continue;
        const int n = len[y], s = stp[y];
        double b0 = 0.0, b1 = 0.0, b2 = 0.0;
        for (int k = 0; k < n; ++k) {
            const double wy = __ldg(&w[(size_t)k * d + y]), wyp = __ldg(&wp[(size_t)k * d + y]);
            const double v0 = a0[(s + k) * kZT + zz], v1 = a1[(s + k) * kZT + zz];
            b0 = fma(wy, v0, b0);
            b1 = fma(wyp, v0, b1);
            b2 = fma(wy, v1, b2);
        }
        const size_t go = ((size_t)xp * d + y) * d + z0 + zz;
        B0[go] = b0;
        B1[go] = b1;
        B2[go] = b2;
    }
}

// stage 3: contract x and finish each voxel.  Block = (y, z tile of ZT/2).
constexpr int kZT3 = 16;
__global__ void __launch_bounds__(256) k_fv_x(const float *src, const FvGeom g, const AxisTables t, const double *B0,
                                              const double *B1, const double *B2, double *data_out, float *data_f32,
                                              float *vec_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int S0 = g.S[0], d = g.d;
    const int y = blockIdx.y, z0 = blockIdx.x * kZT3;
    const int zn = min(kZT3, d - z0);
    double *b0 = (double *)smem;
    double *b1 = b0 + (size_t)S0 * kZT3;
    double *b2 = b1 + (size_t)S0 * kZT3;
    for (int e = threadIdx.x; e < S0 * kZT3; e += blockDim.x) {
        const int xp = e / kZT3, zz = e - xp * kZT3;
        const size_t gi = ((size_t)xp * d + y) * d + z0 + zz;
        const bool ok = zz < zn;
        b0[e] = ok ? B0[gi] : 0.0;
        b1[e] = ok ? B1[gi] : 0.0;
        b2[e] = ok ? B2[gi] : 0.0;
    }
    __syncthreads();
    const int *stp = t.stp, *len = t.len;
    const double *w = t.w, *wp = t.wp;
    for (int o = threadIdx.x; o < d * kZT3; o += blockDim.x) {
        const int x = o / kZT3, zz = o - x * kZT3, z = z0 + zz;
        if (zz >= zn) continue;
        const size_t lin = ((size_t)x * d + y) * d + z;
        // skip tests (VESPER_1_prob_new.py:200-211)
        const int ix = t.idx[x], iy = t.idx[d + y], iz = t.idx[2 * d + z];
        bool valid = ix >= 0 && iy >= 0 && iz >= 0;
        if (valid) valid = src[((size_t)ix * g.S[1] + iy) * g.S[2] + iz] != 0.f;
        double dt = 0.0, px = 0.0, py = 0.0, pz = 0.0;
        if (valid) {
            const int n = len[x], s = stp[x];
            for (int k = 0; k < n; ++k) {
                const double wx = __ldg(&w[(size_t)k * d + x]), wxp = __ldg(&wp[(size_t)k * d + x]);
                const int e = (s + k) * kZT3 + zz;
                dt = fma(wx, b0[e], dt);
                px = fma(wxp, b0[e], px);
                py = fma(wx, b1[e], py);
                pz = fma(wx, b2[e], pz);
            }
        }
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        if (valid && dt != 0.0) {
            // VESPER_1_prob_new.py:242-255
            const double rd = __ddiv_rn(1.0, dt);
            const double t0 = __dsub_rn(__dmul_rn(px, rd), t.pos[x]);
            const double t1 = __dsub_rn(__dmul_rn(py, rd), t.pos[d + y]);
            const double t2 = __dsub_rn(__dmul_rn(pz, rd), t.pos[2 * d + z]);
            double dv = __dadd_rn(__dmul_rn(t0, t0), __dmul_rn(t1, t1));
            dv = __dsqrt_rn(__dadd_rn(dv, __dmul_rn(t2, t2)));
            if (dv == 0.0) dv = 1.0;
            const double rdv = __ddiv_rn(1.0, dv);
            v0 = (float)__dmul_rn(t0, rdv);
            v1 = (float)__dmul_rn(t1, rdv);
            v2 = (float)__dmul_rn(t2, rdv);
        }
        data_out[lin] = dt;
        if (data_f32) data_f32[lin] = (float)dt;
        vec_out[3 * lin + 0] = v0;
        vec_out[3 * lin + 1] = v1;
        vec_out[3 * lin + 2] = v2;
    }
}

// ---- float-float stages ---------------------------------------------------------

// stage 1a.  Blocks below row_blocks list the source rows (xp, yp) that hold a
// non-zero value (a warp per row; 16-byte loads where VEC) and bound each plane's;
// the others list the destination voxels that pass the skip tests
// (VESPER_1_prob_new.py:200-211), mark their columns and zero the rest of the output.
// Lists in any order: every row's and voxel's sums are independent of the others.
// Bound by the read of the source (256^3: 67 MB).
template <bool VEC>
__global__ void __launch_bounds__(256) k_fvf_scan(const float *src, const FvGeom g, const AxisTables t, int row_blocks,
                                                  double *data_out, float *data_f32, float *vec_out) {
    const int S1 = g.S[1], S2 = g.S[2], d = g.d, lane = threadIdx.x & 31;
    if ((int)blockIdx.x < row_blocks) {
        // rounds of 64 rows, 8 per warp, so that a block's rows cost a few atomics
        __shared__ unsigned char flag[64];
        const size_t nrows = (size_t)g.S[0] * S1;
        for (size_t row0 = (size_t)blockIdx.x * 64; row0 < nrows; row0 += (size_t)row_blocks * 64) {
#pragma unroll 2
            for (int q = 0; q < 8; ++q) {
                const size_t row = row0 + (threadIdx.x >> 5) * 8 + q;
                const float *rp = src + row * S2;
                bool nz = false;
                if (row < nrows) {
                    if (VEC) {
#pragma unroll 2
                        for (int e = lane; e < S2 / 4; e += 32) {
                            const float4 v = __ldg((const float4 *)rp + e);
                            nz |= v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f;
                        }
                    } else {
#pragma unroll 4
                        for (int e = lane; e < S2; e += 32) nz |= __ldg(rp + e) != 0.f;
                    }
                }
                nz = __any_sync(0xffffffffu, nz);
                if (lane == 0) flag[(threadIdx.x >> 5) * 8 + q] = nz;
            }
            __syncthreads();
            if (threadIdx.x < 64) {   // two whole warps
                const size_t row = row0 + threadIdx.x;
                const bool nz = flag[threadIdx.x];
                if (row < nrows) t.rowf[row] = nz;
                const unsigned m = __ballot_sync(0xffffffffu, nz);
                int base = 0;
                if (lane == 0 && m) base = atomicAdd(t.count, __popc(m));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (nz) {
                    t.list[base + __popc(m & ((1u << lane) - 1u))] = (int)row;
                    const int xp = (int)(row / S1), yp = (int)(row - (size_t)xp * S1);
                    // the bounds only move outwards: most rows see theirs already there
                    if (yp < *(volatile int *)(t.rlo + xp)) atomicMin(t.rlo + xp, yp);
                    if (yp > *(volatile int *)(t.rhi + xp)) atomicMax(t.rhi + xp, yp);
                    if (xp < *(volatile int *)(t.count + 2)) atomicMin(t.count + 2, xp);
                    if (xp > *(volatile int *)(t.count + 3)) atomicMax(t.count + 3, xp);
                }
            }
            __syncthreads();
        }
        return;
    }
    const int v = ((int)blockIdx.x - row_blocks) * 256 + threadIdx.x, dd = d * d;
    bool valid = false;
    if (v < dd * d) {
        const int x = v / dd, yz = v - x * dd, y = yz / d, z = yz - y * d;
        const int ix = t.idx[x], iy = t.idx[d + y], iz = t.idx[2 * d + z];
        valid = ix >= 0 && iy >= 0 && iz >= 0;
        if (valid) valid = src[((size_t)ix * S1 + iy) * S2 + iz] != 0.f;
        if (valid) {
            t.need[yz] = 1;
        } else {
            data_out[v] = 0.0;
            if (data_f32) data_f32[v] = 0.f;
            vec_out[3 * (size_t)v] = vec_out[3 * (size_t)v + 1] = vec_out[3 * (size_t)v + 2] = 0.f;
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(t.count + 1, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (valid) t.voxels[base + __popc(m & ((1u << lane) - 1u))] = v;
}

// stage 1b (z).  Block b takes listed rows [b kZRows, (b + 1) kZRows): each row's
// non-zero entries are packed in order into shared memory with the count before
// every entry, so that a thread, one output z of one row, sums just the non-zero
// entries of its band (most of a thresholded row is zero, and a zero adds nothing
// to a pair sum).  The z axis's weight pairs are staged too when they fit (SW).
// Every entry of the band for two rows per thread took 101 us (256^3 -> 42^3) and 30
// (128^3 -> 28^3); now 41 and 9.5.  Where the weights are not staged, two loads per entry
// and sum cost more than the zeros once three tenths of a block's entries are not zero:
// such blocks sum every entry of the band for two rows per thread, from one pair of
// weight loads (256^3 -> 128^3, half of the voxels: 958 -> 663 us; zeros
// are the same bits).
constexpr int kZRows = 16;
constexpr int kZThreads = 512;
constexpr int kFfBatch = 8;    // band entries loaded per round by the y stage from global memory
constexpr int kXBatch = 16;    // and by the x stage
struct ZEntry {
    float v;
    int e;
};
// rows: kZRows, fewer where long source rows would not fit
__host__ __device__ inline size_t fvf_z_rows_smem(int S2, int rows) {
    return (size_t)rows * (S2 * sizeof(ZEntry) + (S2 + 1 + 3) / 4 * 4 * sizeof(short));
}
template <bool SW>
__global__ void __launch_bounds__(kZThreads) k_fvf_z(const float *src, const FvGeom g, const AxisTables t, int rows,
                                                     float2 *A0, float2 *A1) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int S2 = g.S[2], d = g.d, WB = g.WB, CN = (S2 + 1 + 3) / 4 * 4;
    const int first = blockIdx.x * rows;
    const int nr = min(rows, t.count[0] - first);
    if (nr <= 0) return;   // block-uniform
    __shared__ int total;  // non-zero entries of the block's rows
    if (!SW && threadIdx.x == 0) total = 0;
    if (!SW) __syncthreads();
    ZEntry *ent = (ZEntry *)smem;                                      // [rows][S2]
    unsigned short *cnt = (unsigned short *)(ent + rows * S2);         // [rows][CN]
    float2 *sw = (float2 *)(smem + fvf_z_rows_smem(S2, rows));         // [WB][d] when SW
    float2 *swp = sw + (SW ? (size_t)WB * d : 0);                      // [WB][d] when SW
    const float2 *gw = t.wf + (size_t)2 * WB * d, *gwp = t.wpf + (size_t)2 * WB * d;
    if (SW)
#pragma unroll 4
        for (int e = threadIdx.x; e < WB * d; e += kZThreads) {
            sw[e] = __ldg(gw + e);
            swp[e] = __ldg(gwp + e);
        }
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < nr; r += kZThreads / 32) {
        const float *rp = src + (size_t)t.list[first + r] * S2;
        int n = 0;
        for (int e0 = 0; e0 < S2; e0 += 32) {
            const int e = e0 + lane;
            const float v = e < S2 ? __ldg(rp + e) : 0.f;
            const unsigned m = __ballot_sync(0xffffffffu, v != 0.f);
            const int at = n + __popc(m & ((1u << lane) - 1u));
            if (e < S2) cnt[r * CN + e] = (unsigned short)at;
            if (v != 0.f) ent[r * S2 + at] = ZEntry{v, e};
            n += __popc(m);
        }
        if (lane == 0) cnt[r * CN + S2] = (unsigned short)n;
        if (!SW && lane == 0) atomicAdd(&total, n);
    }
    __syncthreads();
    const int *stp = t.stp + 2 * d, *len = t.len + 2 * d;
    const float2 *w = SW ? sw : gw, *wp = SW ? swp : gwp;
    if (!SW && total > nr * S2 * 3 / 10) {   // dense rows: every entry, two rows per thread
        float *full = (float *)smem;         // [nr + 1][S2], the last row zero
        __syncthreads();
        for (int e = threadIdx.x; e < (nr + 1) * S2; e += kZThreads) {
            const int r = e / S2;
            full[e] = r < nr ? __ldg(src + (size_t)t.list[first + r] * S2 + (e - r * S2)) : 0.f;
        }
        __syncthreads();
        for (int it = threadIdx.x; it < (nr + 1) / 2 * d; it += kZThreads) {
            const int r = it / d * 2, z = it - r / 2 * d, n = len[z];
            const float *v0 = full + r * S2 + stp[z], *v1 = v0 + S2;
            float s0h[2] = {}, s0l[2] = {}, s1h[2] = {}, s1l[2] = {};
#pragma unroll 2
            for (int k = 0; k < n; ++k) {
                const float2 a = __ldg(w + (size_t)k * d + z), b = __ldg(wp + (size_t)k * d + z);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float v = (u ? v1 : v0)[k];
                    float ph, pl;
                    ff_mul_f(a.x, a.y, v, ph, pl);
                    ff_add(s0h[u], s0l[u], ph, pl);
                    ff_mul_f(b.x, b.y, v, ph, pl);
                    ff_add(s1h[u], s1l[u], ph, pl);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (r + u < nr) {
                    const size_t o = (size_t)t.list[first + r + u] * d + z;
                    A0[o] = make_float2(s0h[u], s0l[u]);
                    A1[o] = make_float2(s1h[u], s1l[u]);
                }
        }
        return;
    }
    for (int it = threadIdx.x; it < nr * d; it += kZThreads) {
        const int r = it / d, z = it - r * d, s = min(stp[z], S2), n = len[z];
        const int lo = cnt[r * CN + s], hi = n > 0 ? cnt[r * CN + s + n] : lo;
        const ZEntry *ep = ent + r * S2;
        const float2 *wz = w + z - (size_t)s * d, *wpz = wp + z - (size_t)s * d;
        float s0h = 0.f, s0l = 0.f, s1h = 0.f, s1l = 0.f;
#pragma unroll 2
        for (int i = lo; i < hi; ++i) {
            const ZEntry q = ep[i];
            const float2 a = wz[(size_t)q.e * d], b = wpz[(size_t)q.e * d];
            float ph, pl;
            ff_mul_f(a.x, a.y, q.v, ph, pl);
            ff_add(s0h, s0l, ph, pl);
            ff_mul_f(b.x, b.y, q.v, ph, pl);
            ff_add(s1h, s1l, ph, pl);
        }
        const size_t o = (size_t)t.list[first + r] * d + z;
        A0[o] = make_float2(s0h, s0l);
        A1[o] = make_float2(s1h, s1l);
    }
}

// stage 2 (y).  Block = (z tile of zw, source plane xp, chunk of yc consecutive
// outputs y).  The rows of A0 and A1 that the chunk's bands cover, between the
// plane's first and last row with a non-zero value (at most rmax, a bound the host
// derives from the geometry), and the chunk's weight pairs are first copied to shared
// memory with coalesced loads that are all in flight together; a block whose rows
// exceed rmax (rmax = 0: the slab does not fit) reads global memory instead, kFfBatch
// band entries per round.  Only the columns that stage 3 will read are computed: the
// block packs them into a list, and each of a column's three sums has a thread (the
// sums are long dependent chains: with three a thread the SMs idled).  A plane without a non-zero value
// gives +0.0, and none before the first such plane or after the last is read.
// All columns, lanes over tiles of 32 z: 79 us (256^3 -> 42^3) and 22 (128^3 -> 28^3);
// now 43 and 18.5.
constexpr int kYThreads = 256;
__global__ void __launch_bounds__(kYThreads) k_fvf_y(const FvGeom g, const AxisTables t, int zw, int yc, int rmax,
                                                     const float2 *A0, const float2 *A1, float2 *B0, float2 *B1,
                                                     float2 *B2) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int ncol;
    const int S1 = g.S[1], d = g.d, WB = g.WB;
    const int z0 = blockIdx.x * zw, xp = blockIdx.y, y0 = blockIdx.z * yc;
    const int yn = min(yc, d - y0), zn = min(zw, d - z0);
    if (xp < t.count[2] || xp > t.count[3] || zn <= 0) return;   // block-uniform, as below
    const int *stp = t.stp + d, *len = t.len + d;
    const float2 *wf = t.wf + (size_t)WB * d, *wpf = t.wpf + (size_t)WB * d;
    const int plo = t.rlo[xp], phi = t.rhi[xp] + 1;
    int r0 = S1, r1 = 0;
    for (int y = y0; y < y0 + yn; ++y) {
        r0 = min(r0, stp[y]);
        r1 = max(r1, stp[y] + len[y]);
    }
    r0 = max(r0, plo);
    r1 = max(min(r1, phi), r0);
    const bool slab = r1 - r0 <= rmax;   // block-uniform
    float2 *s0 = (float2 *)smem;            // [rmax][zw]
    float2 *s1 = s0 + (size_t)rmax * zw;    // [rmax][zw]
    float2 *sw = s1 + (size_t)rmax * zw;    // [yc][WB]
    float2 *swp = sw + (size_t)yc * WB;     // [yc][WB]
    unsigned short *cols = (unsigned short *)(swp + (size_t)yc * WB);   // [yc zw]
    if (threadIdx.x == 0) ncol = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int c0 = 0; c0 < yn * zw; c0 += kYThreads) {
        const int c = c0 + threadIdx.x, yy = c / zw, zz = c - yy * zw;
        const bool on = c < yn * zw && zz < zn && t.need[(y0 + yy) * d + z0 + zz];
        const unsigned m = __ballot_sync(0xffffffffu, on);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&ncol, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (on) cols[base + __popc(m & ((1u << lane) - 1u))] = (unsigned short)c;
    }
    __syncthreads();
    const int nc = ncol;
    if (nc == 0) return;
    if (slab) {
#pragma unroll 4
        for (int e = threadIdx.x; e < (r1 - r0) * zw; e += kYThreads) {
            const int r = e / zw, zz = e - r * zw;
            float2 v0 = make_float2(0.f, 0.f), v1 = v0;
            const size_t row = (size_t)xp * S1 + r0 + r;
            if (zz < zn && t.rowf[row]) {
                v0 = __ldg(A0 + row * d + z0 + zz);
                v1 = __ldg(A1 + row * d + z0 + zz);
            }
            s0[e] = v0;
            s1[e] = v1;
        }
        for (int e = threadIdx.x; e < yn * WB; e += kYThreads) {
            const int k = e / yn, yy = e - k * yn;
            sw[yy * WB + k] = __ldg(wf + (size_t)k * d + y0 + yy);
            swp[yy * WB + k] = __ldg(wpf + (size_t)k * d + y0 + yy);
        }
        __syncthreads();
    }
    // item (sum, column), columns fastest: B0 = sum w A0, B1 = sum wp A0, B2 = sum w A1
    for (int it = threadIdx.x; it < 3 * nc; it += kYThreads) {
        const int q = it >= 2 * nc ? 2 : it >= nc, col = cols[it - q * nc];
        const int yy = col / zw, zz = col - yy * zw, y = y0 + yy, z = z0 + zz;
        const int s = stp[y], k0 = max(0, plo - s), n = min(len[y], phi - s);
        float bh = 0.f, bl = 0.f;
        auto term = [&](float2 w, float2 v) {
            float ph, pl;
            ff_mul(v, w, ph, pl);
            ff_add(bh, bl, ph, pl);
        };
        if (slab) {
            const float2 *a = (q == 2 ? s1 : s0) + (s - r0) * zw + zz;
            const float2 *w = (q == 1 ? swp : sw) + (size_t)yy * WB;
#pragma unroll 4
            for (int k = k0; k < n; ++k) term(w[k], a[k * zw]);
        } else {
            const float2 *w = (q == 1 ? wpf : wf) + y, *A = q == 2 ? A1 : A0;
            const size_t row = (size_t)xp * S1 + s;
            for (int k = k0; k < n; k += kFfBatch) {
                float2 wy[kFfBatch], v[kFfBatch];
#pragma unroll
                for (int u = 0; u < kFfBatch; ++u) {
                    const bool on = k + u < n && t.rowf[row + k + u];
                    const size_t o = (size_t)(k + u) * d;
                    wy[u] = on ? __ldg(w + o) : make_float2(0.f, 0.f);
                    v[u] = on ? __ldg(A + row * d + o + z) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < kFfBatch; ++u) term(wy[u], v[u]);
            }
        }
        (q == 0 ? B0 : q == 1 ? B1 : B2)[((size_t)xp * d + y) * d + z] = make_float2(bh, bl);
    }
}

// The finish of voxel v from its sums D, Px, Py, Pz (VESPER_1_prob_new.py:242-255).
__device__ __forceinline__ void fvf_finish(const AxisTables &t, int d, int v, float2 sd, float2 sx, float2 sy, float2 sz,
                                           double *data_out, float *data_f32, float *vec_out) {
    const int x = v / (d * d), yz = v - x * d * d, y = yz / d, z = yz - y * d;
    const double dt = (double)sd.x + (double)sd.y;
    float o0 = 0.f, o1 = 0.f, o2 = 0.f;
    if (dt != 0.0) {
        const double px = (double)sx.x + (double)sx.y, py = (double)sy.x + (double)sy.y, pz = (double)sz.x + (double)sz.y;
        const double rd = __ddiv_rn(1.0, dt);
        const double t0 = __dsub_rn(__dmul_rn(px, rd), t.pos[x]);
        const double t1 = __dsub_rn(__dmul_rn(py, rd), t.pos[d + y]);
        const double t2 = __dsub_rn(__dmul_rn(pz, rd), t.pos[2 * d + z]);
        double dv = __dadd_rn(__dmul_rn(t0, t0), __dmul_rn(t1, t1));
        dv = __dsqrt_rn(__dadd_rn(dv, __dmul_rn(t2, t2)));
        if (dv == 0.0) dv = 1.0;
        const double rdv = __ddiv_rn(1.0, dv);
        o0 = (float)__dmul_rn(t0, rdv);
        o1 = (float)__dmul_rn(t1, rdv);
        o2 = (float)__dmul_rn(t2, rdv);
    }
    data_out[v] = dt;
    if (data_f32) data_f32[v] = (float)dt;
    vec_out[3 * (size_t)v + 0] = o0;
    vec_out[3 * (size_t)v + 1] = o1;
    vec_out[3 * (size_t)v + 2] = o2;
}

// stage 3 (x) and the finish, four lanes per listed voxel, one for each of its sums
// D, Px, Py, Pz: the column's sums are read along x between the first and last plane
// with a non-zero value, kXBatch entries in flight.  Blocks over all voxels, a slab of
// B0, B1 and B2 in shared memory and 9 of 32 lanes at work took 34 us for 256^3 -> 42^3.
// With the stages above the whole call went from 233 to 121 us there and from 73 to 59
// for 128^3 -> 28^3.
// MANY (grids of kXGrid voxels and more): from kXMany listed voxels on, about 16 warps of
// them per SM, a thread has a voxel and its four sums: a warp's loads then are whole
// lines, and the sums share them (200^3 -> 75^3, every voxel: 172 -> 105 us, a ball 54 ->
// 40).  Smaller grids keep the form for few voxels alone, which is faster without the
// other's registers (100^3 -> 50^3, a ball: 12 us, 15 with them).
constexpr int kXMany = 80000;
constexpr size_t kXGrid = 150000;
constexpr int kXBatch1 = 4;
template <bool MANY>
__global__ void __launch_bounds__(128) k_fvf_x(const FvGeom g, const AxisTables t, const float2 *B0, const float2 *B1,
                                               const float2 *B2, double *data_out, float *data_f32, float *vec_out) {
    const int d = g.d, nv = t.count[1];
    const size_t plane = (size_t)d * d;
    if (MANY && nv >= kXMany) {
        const int i = blockIdx.x * 128 + threadIdx.x;
        if (i >= nv) return;
        const int v = t.voxels[i], x = v / (d * d), yz = v - x * d * d;
        const int s = t.stp[x], k0 = max(0, t.count[2] - s), n = min(t.len[x], t.count[3] + 1 - s);
        const float2 *w = t.wf + x, *wp = t.wpf + x;
        const size_t o = (size_t)s * plane + yz;
        float2 sum[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) sum[q] = make_float2(0.f, 0.f);
        for (int k = k0; k < n; k += kXBatch1) {
            float2 wx[kXBatch1], wxp[kXBatch1], b0[kXBatch1], b1[kXBatch1], b2[kXBatch1];
#pragma unroll
            for (int u = 0; u < kXBatch1; ++u) {
                const int e = min(k + u, n - 1);
                wx[u] = __ldg(w + (size_t)e * d);
                wxp[u] = __ldg(wp + (size_t)e * d);
                b0[u] = __ldg(B0 + o + e * plane);
                b1[u] = __ldg(B1 + o + e * plane);
                b2[u] = __ldg(B2 + o + e * plane);
                if (k + u >= n) b0[u] = b1[u] = b2[u] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kXBatch1; ++u) {
                float ph, pl;
                ff_mul(b0[u], wx[u], ph, pl);
                ff_add(sum[0].x, sum[0].y, ph, pl);
                ff_mul(b0[u], wxp[u], ph, pl);
                ff_add(sum[1].x, sum[1].y, ph, pl);
                ff_mul(b1[u], wx[u], ph, pl);
                ff_add(sum[2].x, sum[2].y, ph, pl);
                ff_mul(b2[u], wx[u], ph, pl);
                ff_add(sum[3].x, sum[3].y, ph, pl);
            }
        }
        fvf_finish(t, d, v, sum[0], sum[1], sum[2], sum[3], data_out, data_f32, vec_out);
        return;
    }
    const int i = blockIdx.x * 32 + (threadIdx.x >> 2), q = threadIdx.x & 3;
    if (blockIdx.x * 32 >= nv) return;
    const int vi = t.voxels[min(i, nv - 1)], xi = vi / (d * d);
    const int s = t.stp[xi], k0 = max(0, t.count[2] - s), n = min(t.len[xi], t.count[3] + 1 - s);
    const float2 *w = (q == 1 ? t.wpf : t.wf) + xi, *b = (q < 2 ? B0 : q == 2 ? B1 : B2) + (size_t)s * plane + vi % (d * d);
    float sh = 0.f, sl = 0.f;
    for (int k = k0; k < n; k += kXBatch) {
        float2 wx[kXBatch], bv[kXBatch];
#pragma unroll
        for (int u = 0; u < kXBatch; ++u) {
            const int e = min(k + u, n - 1);   // every load is made, so that all are in flight
            wx[u] = __ldg(w + (size_t)e * d);
            bv[u] = __ldg(b + (size_t)e * plane);
            if (k + u >= n) bv[u] = make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kXBatch; ++u) {
            float ph, pl;
            ff_mul(bv[u], wx[u], ph, pl);
            ff_add(sh, sl, ph, pl);
        }
    }
    // the finish is float64, at 1/64 of the float32 rate: whole warps of voxels
    __shared__ float2 sums[4][32];
    sums[q][threadIdx.x >> 2] = make_float2(sh, sl);
    __syncthreads();
    const int f = blockIdx.x * 32 + threadIdx.x;
    if (threadIdx.x >= 32 || f >= nv) return;
    fvf_finish(t, d, t.voxels[f], sums[0][threadIdx.x], sums[1][threadIdx.x], sums[2][threadIdx.x], sums[3][threadIdx.x],
               data_out, data_f32, vec_out);
}

// smallest band weight of the geometry (|r| <= fmaxd + 1 on each axis)
static bool fv_float_float(const FvGeom &g) {
    const double r = g.fmaxd + 1.0;
    return std::exp(-1.5 * r * r * g.fsiv) >= 0x1p-70;
}

// The y stage's chunk and slab rows: the chunk's bands cover at most WB +
// floor((c - 1) dw / sw) + 1 source rows (stp is non-decreasing in the output index
// and steps by at most floor(dw / sw) + 1).  About one column of the chunk per
// thread, fewer while the slab exceeds 64 KB (three blocks per SM); rmax = 0 (global
// loads) when even one output's band does not fit.
static void fvf_chunk(const FvGeom &g, int S, int zw, int *c, int *rmax, size_t *bytes) {
    const int want = std::min(g.d, (kYThreads + zw - 1) / zw);
    for (int cc = want; cc >= 1; cc = cc > 1 ? (cc + 1) / 2 : 0) {
        const int r = std::min(S, g.WB + (int)((cc - 1) * g.dw / g.sw) + 2);
        const size_t b = ((size_t)2 * r * zw + 2 * (size_t)cc * g.WB) * sizeof(float2) + (size_t)cc * zw * sizeof(short);
        if (b <= 64 * 1024 || (cc == 1 && b <= 200 * 1024)) {
            *c = cc;
            *rmax = r;
            *bytes = b;
            return;
        }
    }
    *c = 1;
    *rmax = 0;
    *bytes = 2 * (size_t)g.WB * sizeof(float2) + (size_t)zw * sizeof(short);
}

static void fv_geom(int sx, int sy, int sz, double src_width, const double *src_orig, int dim, double dest_width,
                    const double *dest_orig, double dreso, FvGeom *g) {
    g->S[0] = sx;
    g->S[1] = sy;
    g->S[2] = sz;
    g->d = dim;
    g->sw = src_width;
    g->dw = dest_width;
    // VESPER_1_prob_new.py:183-187
    volatile double q = dreso / src_width;
    double fs = q * 0.5;
    fs = fs * fs;
    g->fsiv = 1.0 / fs;
    g->fmaxd = q * 2.0;
    g->WB = (int)(2.0 * g->fmaxd) + 3;
    for (int a = 0; a < 3; ++a) {
        g->sorig[a] = src_orig[a];
        g->dorig[a] = dest_orig[a];
    }
}

static size_t fv_workspace(const FvGeom &g, AxisTables *t, double **A0, double **A1, double **B0, double **B1,
                           double **B2, void *base, size_t cap) {
    Carver cv(base, cap);
    const int d = g.d;
    t->pos = cv.take<double>(3 * (size_t)d);
    t->stp = cv.take<int>(3 * (size_t)d);
    t->len = cv.take<int>(3 * (size_t)d);
    t->idx = cv.take<int>(3 * (size_t)d);
    t->w = cv.take<double>(3 * (size_t)g.WB * d);
    t->wp = cv.take<double>(3 * (size_t)g.WB * d);
    t->wf = cv.take<float2>(3 * (size_t)g.WB * d);
    t->wpf = cv.take<float2>(3 * (size_t)g.WB * d);
    t->rlo = cv.take<int>((size_t)g.S[0]);
    t->rhi = cv.take<int>((size_t)g.S[0]);
    t->list = cv.take<int>((size_t)g.S[0] * g.S[1]);
    t->rowf = cv.take<unsigned char>((size_t)g.S[0] * g.S[1]);
    t->need = cv.take<unsigned char>((size_t)d * d);
    t->voxels = cv.take<int>((size_t)d * d * d);
    t->count = cv.take<int>(4);
    // the partial sums: float64, or float-float pairs of the same 8 bytes
    const size_t rows = (size_t)g.S[0] * g.S[1];
    *A0 = cv.take<double>(rows * d);
    *A1 = cv.take<double>(rows * d);
    *B0 = cv.take<double>((size_t)g.S[0] * d * d);
    *B1 = cv.take<double>((size_t)g.S[0] * d * d);
    *B2 = cv.take<double>((size_t)g.S[0] * d * d);
    return cv.off + 256;
}

}  // namespace vg

using namespace vg;

extern "C" int vesper_fastvec_workspace_size(int sx, int sy, int sz, int dim, size_t *bytes) {
    if (!bytes || sx < 1 || sy < 1 || sz < 1 || dim < 1)
        return fail(VESPER_ERR_INVALID, "vesper_fastvec_workspace_size: bad arguments");
    // the band width depends on dreso / src_width; size for the widest band the
    // caller can ask for below (fmaxd <= 512 source voxels)
    FvGeom g{};
    g.S[0] = sx;
    g.S[1] = sy;
    g.S[2] = sz;
    g.d = dim;
    g.WB = 2 * 512 + 3;
    AxisTables t;
    double *a0, *a1, *b0, *b1, *b2;
    *bytes = fv_workspace(g, &t, &a0, &a1, &b0, &b1, &b2, nullptr, 0);
    return VESPER_OK;
}

extern "C" int vesper_fastvec(const float *src, int sx, int sy, int sz, double src_width, const double *src_orig,
                              int dim, double dest_width, const double *dest_orig, double dreso, double *data_out,
                              float *data_f32, float *vec_out, void *workspace, size_t workspace_bytes,
                              void *stream) {
    if (!src || !src_orig || !dest_orig || !data_out || !vec_out)
        return fail(VESPER_ERR_INVALID, "vesper_fastvec: missing pointer");
    if (sx < 1 || sy < 1 || sz < 1 || dim < 1) return fail(VESPER_ERR_INVALID, "vesper_fastvec: bad sizes");
    if (!(src_width > 0) || !(dreso > 0)) return fail(VESPER_ERR_INVALID, "vesper_fastvec: bad widths");
    FvGeom g;
    fv_geom(sx, sy, sz, src_width, src_orig, dim, dest_width, dest_orig, dreso, &g);
    if (g.fmaxd > 512.0) return fail(VESPER_ERR_UNSUPPORTED, "vesper_fastvec: window %.1f voxels too wide", g.fmaxd);
    AxisTables t;
    double *A0, *A1, *B0, *B1, *B2;
    const size_t need = fv_workspace(g, &t, &A0, &A1, &B0, &B1, &B2, workspace, workspace_bytes);
    if (!workspace || workspace_bytes < need)
        return fail(VESPER_ERR_WORKSPACE, "vesper_fastvec: workspace %zu < %zu bytes", workspace_bytes, need);
    cudaStream_t st = (cudaStream_t)stream;
    k_fv_tables<<<dim3(dim, 3), 128, 0, st>>>(g, t);
    VG_CHECK_LAUNCH("k_fv_tables");
    const size_t nrows = (size_t)sx * sy;
    if (fv_float_float(g)) {
        if ((size_t)17 * sz * sizeof(float) > 200 * 1024)
            return fail(VESPER_ERR_UNSUPPORTED, "vesper_fastvec: source rows too long (%d)", sz);
        float2 *a0 = reinterpret_cast<float2 *>(A0), *a1 = reinterpret_cast<float2 *>(A1);
        float2 *b0 = reinterpret_cast<float2 *>(B0), *b1 = reinterpret_cast<float2 *>(B1),
               *b2 = reinterpret_cast<float2 *>(B2);
        const unsigned row_blocks = (unsigned)std::min<size_t>((nrows + 63) / 64, 1 << 14);
        const size_t vox = (size_t)dim * dim * dim;
        const unsigned vox_blocks = (unsigned)((vox + 255) / 256);
        if (sz % 4 == 0 && ((uintptr_t)src & 15) == 0)
            k_fvf_scan<true><<<row_blocks + vox_blocks, 256, 0, st>>>(src, g, t, (int)row_blocks, data_out, data_f32, vec_out);
        else
            k_fvf_scan<false><<<row_blocks + vox_blocks, 256, 0, st>>>(src, g, t, (int)row_blocks, data_out, data_f32, vec_out);
        VG_CHECK_LAUNCH("k_fvf_scan");
        int rows = kZRows;
        while (rows > 1 && fvf_z_rows_smem(sz, rows) > 64 * 1024) rows /= 2;
        const size_t srows = fvf_z_rows_smem(sz, rows), sweights = 2 * (size_t)g.WB * dim * sizeof(float2);
        const bool zsw = srows + sweights <= 112 * 1024;   // the z weights staged in shared memory, two blocks per SM
        const size_t s1 = srows + (zsw ? sweights : 0);
        const unsigned zb = (unsigned)((nrows + rows - 1) / rows);
        if (zsw) {
            allow_smem(k_fvf_z<true>, s1);
            k_fvf_z<true><<<zb, kZThreads, s1, st>>>(src, g, t, rows, a0, a1);
        } else {
            allow_smem(k_fvf_z<false>, s1);
            k_fvf_z<false><<<zb, kZThreads, s1, st>>>(src, g, t, rows, a0, a1);
        }
        VG_CHECK_LAUNCH("k_fvf_z");
        const int nt = (dim + 31) / 32, zw = (dim + nt - 1) / nt;
        int yc, ry;
        size_t sy2;
        fvf_chunk(g, sy, zw, &yc, &ry, &sy2);
        allow_smem(k_fvf_y, sy2);
        k_fvf_y<<<dim3(nt, sx, (unsigned)((dim + yc - 1) / yc)), kYThreads, sy2, st>>>(g, t, zw, yc, ry, a0, a1, b0, b1, b2);
        VG_CHECK_LAUNCH("k_fvf_y");
        (vox >= kXGrid ? k_fvf_x<true> : k_fvf_x<false>)
            <<<(unsigned)((vox + 31) / 32), 128, 0, st>>>(g, t, b0, b1, b2, data_out, data_f32, vec_out);
        VG_CHECK_LAUNCH("k_fvf_x");
        return VESPER_OK;
    }
    const size_t s1 = (size_t)kRB * sz * sizeof(float);
    if (s1 > 200 * 1024) return fail(VESPER_ERR_UNSUPPORTED, "vesper_fastvec: source rows too long (%d)", sz);
    allow_smem(k_fv_z, s1);
    k_fv_z<<<(unsigned)((nrows + kRB - 1) / kRB), 256, s1, st>>>(src, g, t, A0, A1);
    VG_CHECK_LAUNCH("k_fv_z");
    const size_t s2 = 2 * (size_t)sy * kZT * sizeof(double);
    const size_t s3 = 3 * (size_t)sx * kZT3 * sizeof(double);
    if (s2 > 220 * 1024 || s3 > 220 * 1024)
        return fail(VESPER_ERR_UNSUPPORTED, "vesper_fastvec: source side too large (%d, %d)", sx, sy);
    allow_smem(k_fv_y, s2);
    k_fv_y<<<dim3((dim + kZT - 1) / kZT, sx), 256, s2, st>>>(g, t, A0, A1, B0, B1, B2);
    VG_CHECK_LAUNCH("k_fv_y");
    allow_smem(k_fv_x, s3);
    k_fv_x<<<dim3((dim + kZT3 - 1) / kZT3, dim), 256, s3, st>>>(src, g, t, B0, B1, B2, data_out, data_f32, vec_out);
    VG_CHECK_LAUNCH("k_fv_x");
    return VESPER_OK;
}
