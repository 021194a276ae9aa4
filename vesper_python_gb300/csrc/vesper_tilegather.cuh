// Gather of the rotated query for the register passes of the search: a warp
// fills tiles of 4 packed z lines (8 rows) of one x plane in shared memory.
#pragma once

#include "vesper_passes.cuh"

namespace vg {

// What pass A transforms: the rotated vectors (3 channels), one rotated value,
// the rotated probabilities (4 channels, each masked by itself), or a field
// that is already rotated (the Laplacian mode).
enum SrcKind { kSrcVec = 0, kSrcVal = 1, kSrcProb = 2, kSrcPlain = 3 };
template <int SRC> __host__ __device__ constexpr int src_nch() {
    return SRC == kSrcVec ? 3 : SRC == kSrcProb ? 4 : 1;
}

// First candidate row of destination index t (gather_cands): itself below the
// middle of an odd side, the next one from there on.
template <int D> __device__ __forceinline__ int first_cand(int t) {
    if constexpr ((D & 1) == 0) return t;
    return t + (t >= (D - 1) / 2);
}
template <int D> __device__ __forceinline__ bool has_cand(int t) { return (D & 1) == 0 ? t < D : t < D - 1; }

// Channels of destination (x, y, z) where an axis of an odd side has two candidate
// rows: every candidate's load is issued before the first hit, in the order of
// gather_src (z slowest, x, y fastest; later rows first), is looked for.
// XMID: x is the middle index too.
template <int SRC, int D, bool XMID>
__device__ __forceinline__ void sample_mid(const Src &s, const float (&F)[9], int x, int y, int z, float *out) {
    constexpr float hc = 0.5f * (float)D;
    constexpr int M = (D - 1) / 2, NX = XMID ? 2 : 1, NCH = src_nch<SRC>();
    float4 v[2 * NX * 2];
    bool hit[2 * NX * 2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < NX; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = (a * NX + b) * 2 + e;
                // the second candidate exists at the middle index only
                const bool on = has_cand<D>(x) && has_cand<D>(y) && has_cand<D>(z) && (a == 0 || z == M) &&
                                (b == 0 || x == M) && (e == 0 || y == M);
                int ox, oy, oz;
                hit[k] = on && old_index(F, D, hc, (float)(first_cand<D>(x) - b) - hc, (float)(first_cand<D>(y) - e) - hc,
                                         (float)(first_cand<D>(z) - a) - hc, ox, oy, oz);
                v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!hit[k]) continue;
                const int i = (ox * D + oy) * D + oz;
                if constexpr (SRC == kSrcVec) {
                    v[k] = __ldg(s.q4 + i);
                    hit[k] = v[k].w != 0.f;
                } else if constexpr (SRC == kSrcVal) {
                    v[k].x = __ldg((const float *)s.q4 + i);
                    hit[k] = __ldg(s.data + i) != 0.0;
                } else {
                    v[k] = __ldg(s.p4 + i);
                }
            }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (SRC == kSrcProb) {   // each channel by its own mask
#pragma unroll
        for (int k = 4 * NX - 1; k >= 0; --k) {
            if (v[k].x != 0.f) o.x = v[k].x;
            if (v[k].y != 0.f) o.y = v[k].y;
            if (v[k].z != 0.f) o.z = v[k].z;
            if (v[k].w != 0.f) o.w = v[k].w;
        }
    } else {
#pragma unroll
        for (int k = 4 * NX - 1; k >= 0; --k)
            if (hit[k]) o = v[k];
    }
    if constexpr (SRC == kSrcVec) {
        rotate_vec(F, o.x, o.y, o.z, out);
    } else {
        const float w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int c = 0; c < NCH; ++c) out[c] = w[c];
    }
}

// Rows 2p and 2p + 1 at z of a packed line, without an odd side's middle index.
template <int D>
__device__ __forceinline__ void store_pair(float2 *at, int p, int z, float v0, float v1) {
    if constexpr ((D & 1) != 0) {
        constexpr int M = (D - 1) / 2;
        if (z == M) {
            if (p == M) at->y = 0.f;   // the last line's missing row
            return;
        }
        if (p == M / 2) {
            if constexpr (M % 2)
                at->x = v0;
            else
                at->y = v1;
            return;
        }
    }
    *at = make_float2(v0, v1);
}

// Gather of tile pt of plane x: rows 8 pt .. 8 pt + 7, packed two to a line in
// buf[c][line][pos(z)].  Lanes cover 4 lines x 8 z at a time, so a warp's source voxels
// share cache lines in all three directions.  A voxel with one candidate row per
// axis is one load (its position's x and y terms are kept per row); the voxels
// of an odd side's middle index (3 D^2 of D^3) are left to gather_planes.
// REACH: only the z steps that come within the query's reach are looked at; returns
// whether no voxel of the tile does (nothing is stored then).
template <int SRC, int D, int LS, int CS, bool REACH, class Pos>
__device__ __forceinline__ bool gather_tile(const PassA2 &a, const float (&F)[9], int b, int x, int pt, float2 *buf,
                                            Pos pos) {
    constexpr int NCH = src_nch<SRC>(), NP = (D + 1) / 2, TZ = (D + 7) / 8;
    constexpr int GI = TZ % 3 == 0 ? 3 : TZ % 2 == 0 ? 2 : TZ % 5 == 0 ? 5 : 2;   // z steps whose loads are in flight together
    // half warps take lines 0, 2 and 1, 3: 8 banks apart in the tile layout
    const int lane = threadIdx.x & 31, p = pt * 4 + ((lane >> 2) & 2) + (lane >> 4), zl = lane & 7;
    const bool pon = p < NP;
    float2 *line = buf + p * LS;
    if constexpr (SRC == kSrcPlain) {
        const float *src = a.plain + ((size_t)b * D + x) * (D * D) + 2 * p * D;
#pragma unroll
        for (int t = 0; t < TZ; ++t) {
            const int z = t * 8 + zl;
            if (pon && z < D) line[pos(z)] = make_float2(__ldg(src + z), 2 * p + 1 < D ? __ldg(src + D + z) : 0.f);
        }
        return false;
    } else {
        constexpr float hc = 0.5f * (float)D, df = (float)D;
        const bool xon = has_cand<D>(x);
        const float hx = (float)first_cand<D>(x) - hc;
        float base[2][3];
        bool on[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int y = 2 * p + h;
            on[h] = pon && xon && has_cand<D>(y);
            const float hy = (float)first_cand<D>(y) - hc;
#pragma unroll
            for (int i = 0; i < 3; ++i) base[h][i] = __fmaf_rn(hy, F[i * 3 + 1], __fmul_rn(hx, F[i * 3]));
        }
        int z0 = 0, z1 = D - 1;   // steps outside hold no value
        if constexpr (REACH) {
            // |base + hz c|^2 <= reach, c the matrix's third column: an interval of hz per row.
            // Wide by a voxel for the rounding and one for the first candidates' offset, and
            // only for columns of about unit length, where neither can be more.
            const float r2 = __uint_as_float(__ldg(a.reach + (SRC == kSrcProb))) + 1.f;
            const float cc = F[2] * F[2] + F[5] * F[5] + F[8] * F[8];
            if (cc > 0.5f && cc < 2.f) {
                z0 = D, z1 = -1;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float bc = base[h][0] * F[2] + base[h][1] * F[5] + base[h][2] * F[8];
                    const float bb = base[h][0] * base[h][0] + base[h][1] * base[h][1] + base[h][2] * base[h][2] - r2;
                    const float disc = bc * bc - cc * bb;
                    if (!on[h] || disc < 0.f) continue;
                    const float sq = sqrtf(disc), lo = (-bc - sq) / cc + hc, hi = (-bc + sq) / cc + hc;
                    z0 = min(z0, (int)fminf(fmaxf(lo, 0.f), df) - 3);
                    z1 = max(z1, (int)fminf(fmaxf(hi, -4.f), df) + 2);
                }
                z0 = __reduce_min_sync(0xffffffffu, z0);
                z1 = __reduce_max_sync(0xffffffffu, z1);
                // the tile of an odd side's middle row has voxels of another row's position
                if (z0 > z1 && ((D & 1) == 0 || pt != (D - 1) / 16)) return true;
            }
        }
#pragma unroll 1
        for (int t0 = 0; t0 < TZ; t0 += GI) {
            if (REACH && (t0 * 8 > z1 || (t0 + GI) * 8 <= z0)) {
#pragma unroll
                for (int g = 0; g < GI; ++g) {
                    const int z = (t0 + g) * 8 + zl;
                    if (pon && z < D)
#pragma unroll
                        for (int c = 0; c < NCH; ++c) store_pair<D>(line + c * CS + pos(z), p, z, 0.f, 0.f);
                }
                continue;
            }
            int src[GI][2];
#pragma unroll
            for (int g = 0; g < GI; ++g) {
                const int z = (t0 + g) * 8 + zl;
                const bool zon = has_cand<D>(z);
                const float hz = (float)first_cand<D>(z) - hc;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float o0 = __fadd_rn(__fmaf_rn(hz, F[2], base[h][0]), hc);
                    const float o1 = __fadd_rn(__fmaf_rn(hz, F[5], base[h][1]), hc);
                    const float o2 = __fadd_rn(__fmaf_rn(hz, F[8], base[h][2]), hc);
                    const bool in = on[h] && zon && o0 >= 0.f && o1 >= 0.f && o2 >= 0.f && o0 < df && o1 < df && o2 < df;
                    src[g][h] = in ? ((int)o0 * D + (int)o1) * D + (int)o2 : -1;
                }
            }
            if constexpr (SRC == kSrcVal) {
                float v[GI][2];
#pragma unroll
                for (int g = 0; g < GI; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        v[g][h] = src[g][h] >= 0 ? __ldg((const float *)a.src.q4 + src[g][h]) : 0.f;
#pragma unroll
                for (int g = 0; g < GI; ++g) {
                    const int z = (t0 + g) * 8 + zl;
                    if (pon && z < D) store_pair<D>(line + pos(z), p, z, v[g][0], v[g][1]);
                }
            } else {
                const float4 *q = SRC == kSrcVec ? a.src.q4 : a.src.p4;
                float4 v[GI][2];
#pragma unroll
                for (int g = 0; g < GI; ++g)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        v[g][h] = src[g][h] >= 0 ? __ldg(q + src[g][h]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int g = 0; g < GI; ++g) {
                    const int z = (t0 + g) * 8 + zl;
                    float r[2][NCH];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 w = v[g][h];
                        if constexpr (SRC == kSrcVec) {
                            rotate_vec(F, w.x, w.y, w.z, r[h]);
                        } else {
                            r[h][0] = w.x;
                            r[h][1] = w.y;
                            r[h][2] = w.z;
                            r[h][3] = w.w;
                        }
                    }
                    if (pon && z < D)
#pragma unroll
                        for (int c = 0; c < NCH; ++c) store_pair<D>(line + c * CS + pos(z), p, z, r[0][c], r[1][c]);
                }
            }
        }
    }
    return false;
}

// Gather of pn planes from x0 by a CTA of NW warps, each into tiles of its own (plane
// stride: the source's channels times CS); on an odd side the voxels of the middle
// index are shared out over the whole CTA first (2 D - 1 of a plane, or all of the
// middle plane and the row that its last line lacks).  Ready after a block barrier.
// REACH (a tile per warp): whether the warp's tile holds no value and is unwritten.
template <int SRC, int D, int LS, int CS, int NW, bool REACH, class Pos>
__device__ __forceinline__ bool gather_planes(const PassA2 &a, const float (&F)[9], int b, int x0, int pn, float2 *buf,
                                              Pos pos) {
    constexpr int NCH = src_nch<SRC>(), TP = ((D + 1) / 2 + 3) / 4;
    if constexpr (SRC == kSrcVec) {
        // a matrix that is not finite puts no voxel on the grid; its product with the
        // zeros of the missing voxels must not reach the plane
        bool finite = true;
#pragma unroll
        for (int i = 0; i < 9; ++i) finite = finite && fabsf(F[i]) <= 3.4028234e38f;
        if (!finite) {
            for (int e = threadIdx.x; e < pn * 3 * CS; e += NW * 32) buf[e] = make_float2(0.f, 0.f);
            return false;
        }
    }
    if constexpr ((D & 1) != 0 && SRC != kSrcPlain) {
        constexpr int M = (D - 1) / 2;
        auto put = [&](int pl, int y, int z, const float *o) {
#pragma unroll
            for (int c = 0; c < NCH; ++c) ((float *)(buf + (pl * NCH + c) * CS + (y >> 1) * LS + pos(z)))[y & 1] = o[c];
        };
        float o[NCH];
#pragma unroll 1
        for (int e = threadIdx.x; e < pn * (2 * D - 1); e += NW * 32) {
            const int pl = e / (2 * D - 1), f = e - pl * (2 * D - 1);
            if (x0 + pl == M) continue;
            const int y = f < D ? M : f - D + (f - D >= M), z = f < D ? f : M;
            sample_mid<SRC, D, false>(a.src, F, x0 + pl, y, z, o);
            put(pl, y, z, o);
        }
        if (M >= x0 && M < x0 + pn)
#pragma unroll 1
            for (int e = threadIdx.x; e < D * (D + 1); e += NW * 32) {
                sample_mid<SRC, D, true>(a.src, F, M, e / D, e % D, o);
                put(M - x0, e / D, e % D, o);
            }
    }
    bool empty = false;
    for (int pt = threadIdx.x >> 5; pt < pn * TP; pt += NW) {
        const int pl = pt / TP, x = x0 + pl;
        if ((D & 1) != 0 && SRC != kSrcPlain && x == (D - 1) / 2) continue;
        empty = gather_tile<SRC, D, LS, CS, REACH>(a, F, b, x, pt - pl * TP, buf + pl * NCH * CS, pos);
    }
    return empty;
}

}  // namespace vg
