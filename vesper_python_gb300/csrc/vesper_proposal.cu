// Learned rotation proposal: a small 3-D convolutional encoder applied to the
// target and the query vector fields, a rotational correlation of the two
// feature fields at zero translation over the angle grid, and the kernels to
// train it (backward passes, softmax cross-entropy, Adam).  Nothing in the
// reference corresponds to this: it orders the rotation grid so that only its
// best-scored fraction is correlated by vesper_search.
//
// Layouts: activations [C][d][d][d] float32 (channel-major); weights
// [Cout][Cin][27] stored as bfloat16 (3x3x3 taps, z fastest) with float32
// accumulation; biases float32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>

#include "vesper_common.cuh"

namespace vg {

// blocks of the score backward pass (two waves of the 152 SMs at most); each
// keeps its partial gradients in shared memory and writes them to its own
// workspace slot
constexpr int kPropBlocks = 304;
constexpr int kPropSMs = 152;

// ---- convolution (3x3x3, zero padding) ----------------------------------------
__global__ void k_conv_fwd(const float *in, int cin, const __nv_bfloat16 *W, const float *bias, int cout, int d,
                           int relu, float *out) {
    const int n = d * d * d;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int co = blockIdx.y;
    in += (size_t)blockIdx.z * cin * n;     // map blockIdx.z of a stack
    out += (size_t)blockIdx.z * cout * n;
    if (v >= n) return;
    const int x = v / (d * d), y = (v / d) % d, z = v % d;
    float acc = bias ? bias[co] : 0.f;
    const __nv_bfloat16 *w = W + (size_t)co * cin * 27;
    for (int ci = 0; ci < cin; ++ci) {
        const float *src = in + (size_t)ci * n;
        const __nv_bfloat16 *wc = w + ci * 27;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const int xx = x + o / 9 - 1, yy = y + (o / 3) % 3 - 1, zz = z + o % 3 - 1;
            if (xx < 0 || yy < 0 || zz < 0 || xx >= d || yy >= d || zz >= d) continue;
            acc = fmaf(__bfloat162float(wc[o]), src[(xx * d + yy) * d + zz], acc);
        }
    }
    out[(size_t)co * n + v] = relu ? fmaxf(acc, 0.f) : acc;
}

// Quotients by a small divisor through the high half of a product: m = recip(d);
// exact for v d < 2^32.
__host__ __device__ __forceinline__ unsigned recip(unsigned d) { return 0xffffffffu / d + 1u; }
__device__ __forceinline__ int quot(int v, int d, unsigned m) { return d == 1 ? v : (int)__umulhi((unsigned)v, m); }

// Four output channels of one voxel (w: [cin][27][4], as k_conv_s stages them), in the order
// of k_conv_fwd; a call of its own, so that it takes no registers where it is not made.
__device__ __noinline__ void conv_voxel(const float *in, int cin, const float4 *w, const float *bias, int d, int relu, int v,
                                        float *out) {
    const int n = d * d * d, x = v / (d * d), y = v / d % d, z = v % d;
    float4 a = bias ? make_float4(bias[0], bias[1], bias[2], bias[3]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int t = 0; t < cin * 27; ++t) {
        const int o = t % 27, xx = x + o / 9 - 1, yy = y + o / 3 % 3 - 1, zz = z + o % 3 - 1;
        if (xx < 0 || yy < 0 || zz < 0 || xx >= d || yy >= d || zz >= d) continue;
        const float f = in[(size_t)(t / 27) * n + (xx * d + yy) * d + zz];
        a = make_float4(fmaf(w[t].x, f, a.x), fmaf(w[t].y, f, a.y), fmaf(w[t].z, f, a.z), fmaf(w[t].w, f, a.w));
    }
    out[v] = relu ? fmaxf(a.x, 0.f) : a.x;
    out[n + v] = relu ? fmaxf(a.y, 0.f) : a.y;
    out[2 * n + v] = relu ? fmaxf(a.z, 0.f) : a.z;
    out[3 * n + v] = relu ? fmaxf(a.w, 0.f) : a.w;
}

// The same layer, and its input gradient, with 4 output channels and ZS consecutive z
// voxels per thread: the 4 channels' weights sit in shared memory as float32 in
// [summed channel][27][4] order (a tap's four weights are one 16-byte broadcast), and
// a summed channel's 9 (x, y) neighbour rows of ZS + 2 values are loaded together,
// zero off the grid, before any product, so a channel costs one load latency instead
// of one per row behind its bounds test (the four layers of two side-15 maps 490 -> 150
// us, of 16 maps 460 -> 290).  Sums in the order of k_conv_fwd (bias, then channel,
// then tap) and of k_conv_bwd_data (channel, then tap); a tap off the grid adds +-0, so
// results are the same bits for finite weights.  Forward, a voxel whose sums are not
// finite is summed again by conv_voxel, which leaves such taps out as k_conv_fwd does (32
// -> 32 channels, 16 maps of side 15: 119.5 and 121.5 us, side 18 234 and 216).  Backward a
// weight that is not finite gives NaN at the border, where k_conv_bwd_data has none: that
// kernel's registers would cost its layers up to 30 % (side 15 76 -> 99 us).
// BWD: the sums run over the layer's output channels (their gradient masked where a
// ReLU let nothing through) and the taps are mirrored.
// SPL: a block's warps share 32 threads' voxels and sum nin / SPL channels each (added
// in warp order), where a layer has too few voxels to hide a warp's latencies.
template <int ZS, bool BWD, int SPL>
__global__ void __launch_bounds__(128) k_conv_s(const float *in, const float *mask, int nin, const __nv_bfloat16 *W,
                                                const float *bias, int nout, int d, int relu, float *out) {
    extern __shared__ float4 wsh4[];   // [nin][27]
    float *wsh = (float *)wsh4;
    const int n = d * d * d, nzs = (d + ZS - 1) / ZS, c0 = blockIdx.y * 4;
    in += (size_t)blockIdx.z * nin * n;     // map blockIdx.z of a stack
    out += (size_t)blockIdx.z * nout * n;
    for (int e = threadIdx.x; e < 4 * nin * 27; e += blockDim.x) {
        const int j = e & 3, o = (e >> 2) % 27, c = (e >> 2) / 27;
        wsh[e] = __bfloat162float(BWD ? W[((size_t)c * nout + c0 + j) * 27 + o] : W[((size_t)(c0 + j) * nin + c) * 27 + o]);
    }
    __syncthreads();
    const int split = SPL > 1 ? threadIdx.x / (128 / SPL) : 0;
    const int u = blockIdx.x * (128 / SPL) + (SPL > 1 ? threadIdx.x % (128 / SPL) : threadIdx.x);
    if (SPL == 1 && u >= d * d * nzs) return;
    const int x = u / (d * nzs), y = (u / nzs) % d, z0 = (u % nzs) * ZS;   // x >= d past the end: each row is tested, nothing is stored
    // the 9 rows' places and the z values on the grid, a bit each
    unsigned rows = 0u, zs = 0u;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        const int xx = x + r / 3 - 1, yy = y + r % 3 - 1;
        rows |= (unsigned)(xx >= 0 && xx < d && yy >= 0 && yy < d) << r;
    }
#pragma unroll
    for (int e = 0; e < ZS + 2; ++e) zs |= (unsigned)(z0 + e - 1 >= 0 && z0 + e - 1 < d) << e;
    const int at = ((x - 1) * d + y - 1) * d + z0 - 1;
    float acc[ZS][4];
#pragma unroll
    for (int i = 0; i < ZS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = !BWD && bias && split == 0 ? bias[c0 + j] : 0.f;
    const int per = (nin + SPL - 1) / SPL, c1 = min(nin, (split + 1) * per);
#pragma unroll(ZS == 1 && !BWD ? 2 : 1)
    for (int c = split * per; c < c1; ++c) {
        const float *src = in + (size_t)c * n + at;
        float v[9][ZS + 2];
#pragma unroll
        for (int r = 0; r < 9; ++r)
#pragma unroll
            for (int e = 0; e < ZS + 2; ++e)
                v[r][e] = (rows >> r & 1u) && (zs >> e & 1u) ? __ldg(src + (r / 3 * d + r % 3) * d + e) : 0.f;
        if (BWD && mask) {
            const float *mk = mask + (size_t)c * n + at;
#pragma unroll
            for (int r = 0; r < 9; ++r)
#pragma unroll
                for (int e = 0; e < ZS + 2; ++e)
                    if ((rows >> r & 1u) && (zs >> e & 1u) && !(__ldg(mk + (r / 3 * d + r % 3) * d + e) > 0.f))
                        v[r][e] = 0.f;
        }
        const float4 *w = wsh4 + (size_t)c * 27;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const float4 w4 = w[o];
#pragma unroll
            for (int i = 0; i < ZS; ++i) {
                const float t = v[BWD ? 8 - o / 3 : o / 3][i + (BWD ? 2 - o % 3 : o % 3)];
                acc[i][0] = fmaf(w4.x, t, acc[i][0]);
                acc[i][1] = fmaf(w4.y, t, acc[i][1]);
                acc[i][2] = fmaf(w4.z, t, acc[i][2]);
                acc[i][3] = fmaf(w4.w, t, acc[i][3]);
            }
        }
    }
    unsigned odd = 0u;   // voxels whose sums are not finite
    if (SPL > 1) {
        static_assert(SPL == 1 || ZS == 1, "split channels: one voxel per thread");
        __shared__ float part[SPL][128 / SPL][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) part[split][threadIdx.x % (128 / SPL)][j] = acc[0][j];
        __syncthreads();
        if (split || u >= n) return;
#pragma unroll
        for (int s = 1; s < SPL; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][j] += part[s][threadIdx.x][j];
    }
#pragma unroll
    for (int i = 0; i < ZS; ++i) {
        const int z = z0 + i;
        if (z >= d) break;
        const size_t v = ((size_t)x * d + y) * d + z;
#pragma unroll
        for (int j = 0; j < 4; ++j) out[(size_t)(c0 + j) * n + v] = !BWD && relu ? fmaxf(acc[i][j], 0.f) : acc[i][j];
        if (!BWD && !(fabsf(acc[i][0]) + fabsf(acc[i][1]) + fabsf(acc[i][2]) + fabsf(acc[i][3]) <= FLT_MAX)) odd |= 1u << i;
    }
    if constexpr (!BWD)
#pragma unroll 1
        for (; odd; odd &= odd - 1)
            conv_voxel(in, nin, wsh4, bias ? bias + c0 : nullptr, d, relu, (x * d + y) * d + z0 + __ffs(odd) - 1,
                       out + (size_t)c0 * n);
}

// Launch, or false where the weights do not fit or the channels do not group.
// 4 voxels per thread; a few maps leave most SMs without a block then: one voxel
// each, backwards with the channels split over the block's warps.
template <bool BWD>
static bool conv_s(const float *in, const float *mask, const __nv_bfloat16 *W, const float *bias, int nin, int nout, int d,
                   int relu, int nmap, float *out, cudaStream_t st) {
    const size_t sm = (size_t)4 * nin * 27 * sizeof(float);
    if (nout % 4 || sm + 4096 > (size_t)smem_limit()) return false;
    const int n = d * d * d, nu = d * d * ((d + 3) / 4);
    if ((long long)((nu + 127) / 128) * (nout / 4) * nmap < 2 * kPropSMs) {
        constexpr int SPL = BWD ? 4 : 1;   // the forward keeps k_conv_fwd's order of sums
        allow_smem(k_conv_s<1, BWD, SPL>, sm);
        k_conv_s<1, BWD, SPL><<<dim3((n + 128 / SPL - 1) / (128 / SPL), nout / 4, nmap), 128, sm, st>>>(
            in, mask, nin, W, bias, nout, d, relu, out);
    } else {
        allow_smem(k_conv_s<4, BWD, 1>, sm);
        k_conv_s<4, BWD, 1><<<dim3((nu + 127) / 128, nout / 4, nmap), 128, sm, st>>>(in, mask, nin, W, bias, nout, d, relu,
                                                                                     out);
    }
    return true;
}

// din[ci][v] = sum_co sum_o W[co][ci][o] * g[co][v - o],  g = dout (masked by
// out > 0 for a ReLU layer)
__global__ void k_conv_bwd_data(const float *dout, const float *out, int relu, const __nv_bfloat16 *W, int cin,
                                int cout, int d, float *din) {
    const int n = d * d * d;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int ci = blockIdx.y;
    if (v >= n) return;
    const int x = v / (d * d), y = (v / d) % d, z = v % d;
    float acc = 0.f;
    for (int co = 0; co < cout; ++co) {
        const float *g = dout + (size_t)co * n;
        const float *o_ = out + (size_t)co * n;
        const __nv_bfloat16 *wc = W + ((size_t)co * cin + ci) * 27;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const int xx = x - (o / 9 - 1), yy = y - ((o / 3) % 3 - 1), zz = z - (o % 3 - 1);
            if (xx < 0 || yy < 0 || zz < 0 || xx >= d || yy >= d || zz >= d) continue;
            const int u = (xx * d + yy) * d + zz;
            const float gv = (relu && !(o_[u] > 0.f)) ? 0.f : g[u];
            acc = fmaf(__bfloat162float(wc[o]), gv, acc);
        }
    }
    din[(size_t)ci * n + v] = acc;
}

// dW[co][ci][o] += sum_v g[co][v] * in[ci][v + o]; db[co] += sum_v g[co][v].
// One block per (co, ci); 27 taps reduced over the voxels.
__global__ void k_conv_bwd_weight(const float *dout, const float *out, int relu, const float *in, int cin, int cout,
                                  int d, float *dW, float *db) {
    const int n = d * d * d;
    const int co = blockIdx.x / cin, ci = blockIdx.x % cin;
    __shared__ float red[28][32];
    float acc[28];
#pragma unroll
    for (int o = 0; o < 28; ++o) acc[o] = 0.f;
    const float *g = dout + (size_t)co * n;
    const float *o_ = out + (size_t)co * n;
    const float *src = in + (size_t)ci * n;
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        const float gv = (relu && !(o_[v] > 0.f)) ? 0.f : g[v];
        if (gv == 0.f) continue;
        const int x = v / (d * d), y = (v / d) % d, z = v % d;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const int xx = x + o / 9 - 1, yy = y + (o / 3) % 3 - 1, zz = z + o % 3 - 1;
            if (xx < 0 || yy < 0 || zz < 0 || xx >= d || yy >= d || zz >= d) continue;
            acc[o] = fmaf(gv, src[(xx * d + yy) * d + zz], acc[o]);
        }
        acc[27] += gv;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 0; o < 28; ++o) {
        float s = acc[o];
        for (int k = 16; k > 0; k >>= 1) s += __shfl_down_sync(0xffffffffu, s, k);
        if (lane == 0) red[o][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < 28) {
        float s = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
        if (threadIdx.x < 27)
            dW[((size_t)co * cin + ci) * 27 + threadIdx.x] += s;
        else if (ci == 0)
            db[co] += s;
    }
}

// The same weight gradients with kWgCo output channels per block: the input channel
// sits in shared memory with a zero border, so a voxel's 27 neighbours are plain
// loads, each used for kWgCo products, where one block per (co, ci) pair spent its
// instructions on the neighbours' bounds (the eight layers of a training step at side 15
// 354 -> 237 us).  2 channels and 256 threads: 4 channels take 192 registers.
// The products with the border and with zero gradients, which k_conv_bwd_weight leaves
// out, add zeros: the same sums for finite values.  A block whose sums are not finite
// makes them again without.
constexpr int kWgCo = 2;
constexpr int kWgThreads = 256;
__global__ void __launch_bounds__(kWgThreads) k_conv_bwd_weight_s(const float *dout, const float *out, int relu,
                                                                  const float *in, int cin, int cout, int d, float *dW,
                                                                  float *db, unsigned md, unsigned mp) {
    extern __shared__ float pad[];   // [d + 2]^3
    __shared__ float red[kWgThreads / 32][kWgCo * 28];
    const int n = d * d * d, p = d + 2;
    const int ci = blockIdx.x % cin, co0 = blockIdx.x / cin * kWgCo;
    const float *src = in + (size_t)ci * n;
    for (int e = threadIdx.x; e < p * p * p; e += kWgThreads) {
        const int q = quot(e, p, mp), x = quot(q, p, mp) - 1, y = q - (x + 1) * p - 1, z = e - q * p - 1;
        const bool on = x >= 0 && y >= 0 && z >= 0 && x < d && y < d && z < d;
        pad[e] = on ? __ldg(src + (x * d + y) * d + z) : 0.f;
    }
    __syncthreads();
    float acc[kWgCo][28];
#pragma unroll
    for (int j = 0; j < kWgCo; ++j)
#pragma unroll
        for (int o = 0; o < 28; ++o) acc[j][o] = 0.f;
#pragma unroll 4
    for (int v = threadIdx.x; v < n; v += kWgThreads) {
        float g[kWgCo];
#pragma unroll
        for (int j = 0; j < kWgCo; ++j) {
            const size_t i = (size_t)(co0 + j) * n + v;
            g[j] = __ldg(dout + i);
            if (relu && !(__ldg(out + i) > 0.f)) g[j] = 0.f;
            acc[j][27] += g[j];
        }
        const int q = quot(v, d, md), x = quot(q, d, md);
        const float *c = pad + (x * p + q - x * d) * p + v - q * d;
#pragma unroll
        for (int o = 0; o < 27; ++o) {
            const float t = c[(o / 9 * p + o / 3 % 3) * p + o % 3];
#pragma unroll
            for (int j = 0; j < kWgCo; ++j) acc[j][o] = fmaf(g[j], t, acc[j][o]);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < kWgCo; ++j)
#pragma unroll
        for (int o = 0; o < 28; ++o) {
            float t = acc[j][o];
            for (int k = 16; k > 0; k >>= 1) t += __shfl_down_sync(0xffffffffu, t, k);
            if (lane == 0) red[warp][j * 28 + o] = t;
        }
    __syncthreads();
    const int e = threadIdx.x;
    auto total = [&]() {
        float t = 0.f;
        if (e < kWgCo * 28)
            for (int w = 0; w < kWgThreads / 32; ++w) t += red[w][e];
        return t;
    };
    float t = total();
    if (__syncthreads_or(!(fabsf(t) <= FLT_MAX))) {
        // once more, one sum after another, without the products that k_conv_bwd_weight
        // leaves out: of a zero gradient, and off the grid
#pragma unroll 1
        for (int f = 0; f < kWgCo * 28; ++f) {
            const int o = f % 28, ox = o / 9, oy = o / 3 % 3, oz = o % 3;
            float a = 0.f;
#pragma unroll 1
            for (int v = threadIdx.x; v < n; v += kWgThreads) {
                const size_t i = (size_t)(co0 + f / 28) * n + v;
                const float g = relu && !(__ldg(out + i) > 0.f) ? 0.f : __ldg(dout + i);
                const int x = v / (d * d) + ox, y = v / d % d + oy, z = v % d + oz;   // in pad
                if (o == 27)
                    a += g;
                else if (g != 0.f && x >= 1 && y >= 1 && z >= 1 && x <= d && y <= d && z <= d)
                    a = fmaf(g, pad[(x * p + y) * p + z], a);
            }
            for (int k = 16; k > 0; k >>= 1) a += __shfl_down_sync(0xffffffffu, a, k);
            if (lane == 0) red[warp][f] = a;
        }
        __syncthreads();
        t = total();
    }
    if (e >= kWgCo * 28) return;
    const int j = e / 28, o = e % 28;
    if (o < 27)
        dW[((size_t)(co0 + j) * cin + ci) * 27 + o] += t;
    else if (ci == 0)
        db[co0 + j] += t;
}

// ---- network input ---------------------------------------------------------------
// out[c][X][Y][Z], c = (vx, vy, vz, mask = data != 0), each the mean over the
// pool^3 block of voxels (pool X .. pool X + pool - 1, clipped at the grid
// edge) of the fastVEC output of one map.
__global__ void k_prop_field(const double *data, const float *vec, int d, int pool, int dp, float *out) {
    const int np = dp * dp * dp;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const int X = i / (dp * dp), Y = (i / dp) % dp, Z = i % dp;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    int cnt = 0;
    for (int x = X * pool; x < min(d, X * pool + pool); ++x)
        for (int y = Y * pool; y < min(d, Y * pool + pool); ++y)
            for (int z = Z * pool; z < min(d, Z * pool + pool); ++z) {
                const size_t v = ((size_t)x * d + y) * d + z;
                acc[0] += vec[3 * v];
                acc[1] += vec[3 * v + 1];
                acc[2] += vec[3 * v + 2];
                acc[3] += data[v] != 0.0 ? 1.f : 0.f;
                ++cnt;
            }
    const float inv = 1.f / (float)cnt;
#pragma unroll
    for (int c = 0; c < 4; ++c) out[(size_t)c * np + i] = acc[c] * inv;
}

// ---- rotational correlation at zero translation --------------------------------
// Source voxel of destination v under rotation F: the reference's gather rule
// (gather_src) with every in-bounds voxel accepted.
__device__ __forceinline__ int prop_src(const float *F, int d, int v) {
    const int x = v / (d * d), y = (v / d) % d, z = v % d;
    return gather_src(F, d, x, y, z, [](int) { return true; });
}

// s[r] = sum_v sum_k ET[k][v] * EQ[k][src_r(v)]; one block per rotation.
__global__ void k_prop_score(const float *ET, const float *EQ, int K, int d, const float *rotmats, int nrot,
                             float *scores) {
    __shared__ float F[9];
    __shared__ float red[32];
    const int r = blockIdx.x;
    if (threadIdx.x < 9) F[threadIdx.x] = rotmats[(size_t)r * 9 + threadIdx.x];
    __syncthreads();
    const int n = d * d * d;
    float acc = 0.f;
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        const int s = prop_src(F, d, v);
        if (s < 0) continue;
        for (int k = 0; k < K; ++k) acc = fmaf(ET[(size_t)k * n + v], EQ[(size_t)k * n + s], acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        scores[r] = s;
    }
}

// [nmap][K][n] -> [nmap][n][K]
__global__ void k_vmajor(const float *in, int K, int n, float *out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t per = (size_t)K * n;
    if (i >= per) return;
    const size_t m = blockIdx.y;
    const int v = (int)(i / K), k = (int)(i % K);
    out[m * per + i] = in[m * per + (size_t)k * n + v];
}

// The same scores from voxel-major features (K a multiple of 4): one voxel's
// K channels are K/4 float4 loads, so the gathered query voxel costs whole
// 32-byte sectors instead of K scattered words.
template <int K4>
__global__ void k_prop_score_vm(const float4 *ET, const float4 *EQ, int d, const float *rotmats, float *scores) {
    __shared__ float F[9];
    __shared__ float red[32];
    const int r = blockIdx.x;
    if (threadIdx.x < 9) F[threadIdx.x] = rotmats[(size_t)r * 9 + threadIdx.x];
    __syncthreads();
    const int n = d * d * d;
    float acc = 0.f;
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        const int s = prop_src(F, d, v);
        if (s < 0) continue;
#pragma unroll
        for (int j = 0; j < K4; ++j) {
            const float4 a = __ldg(ET + (size_t)v * K4 + j), b = __ldg(EQ + (size_t)s * K4 + j);
            acc = fmaf(a.x, b.x, acc);
            acc = fmaf(a.y, b.y, acc);
            acc = fmaf(a.z, b.z, acc);
            acc = fmaf(a.w, b.w, acc);
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        scores[r] = t;
    }
}

// [nmap][K][n] float32 -> [nmap][n][K] float16 (the inference features)
__global__ void k_vmajor_f16(const float *in, int K, int n, __half *out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t per = (size_t)K * n;
    if (i >= per) return;
    const size_t m = blockIdx.y;
    const int v = (int)(i / K), k = (int)(i % K);
    out[m * per + i] = __float2half_rn(in[m * per + (size_t)k * n + (size_t)v]);
}

// Scores of RPB rotations per block from float16 voxel-major features, K8
// groups of 8 channels (one 16-byte load per voxel and group): each target
// voxel's features are loaded once for the block's RPB rotations, the
// gathered query voxel once per rotation; products accumulate in float32.
template <int K8, int RPB>
__global__ void __launch_bounds__(256) k_prop_score_f16(const uint4 *ET, const uint4 *EQ, int d,
                                                        const float *rotmats, int nrot, float *scores) {
    __shared__ float F[RPB][9];
    __shared__ float red[RPB][32];
    const int r0 = blockIdx.x * RPB;
    if (threadIdx.x < 9 * RPB) {
        const int j = threadIdx.x / 9, e = threadIdx.x % 9;
        F[j][e] = r0 + j < nrot ? rotmats[(size_t)(r0 + j) * 9 + e] : 0.f;
    }
    __syncthreads();
    const int n = d * d * d;
    float acc[RPB];
#pragma unroll
    for (int j = 0; j < RPB; ++j) acc[j] = 0.f;
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        float2 t[K8][4];
#pragma unroll
        for (int g = 0; g < K8; ++g) {
            const uint4 a = __ldg(ET + (size_t)v * K8 + g);
            t[g][0] = __half22float2(*(const __half2 *)&a.x);
            t[g][1] = __half22float2(*(const __half2 *)&a.y);
            t[g][2] = __half22float2(*(const __half2 *)&a.z);
            t[g][3] = __half22float2(*(const __half2 *)&a.w);
        }
#pragma unroll
        for (int j = 0; j < RPB; ++j) {
            if (r0 + j >= nrot) break;
            const int s = prop_src(F[j], d, v);
            if (s < 0) continue;
#pragma unroll
            for (int g = 0; g < K8; ++g) {
                const uint4 b = __ldg(EQ + (size_t)s * K8 + g);
                const float2 q0 = __half22float2(*(const __half2 *)&b.x), q1 = __half22float2(*(const __half2 *)&b.y);
                const float2 q2 = __half22float2(*(const __half2 *)&b.z), q3 = __half22float2(*(const __half2 *)&b.w);
                float a = acc[j];
                a = fmaf(t[g][0].x, q0.x, a);
                a = fmaf(t[g][0].y, q0.y, a);
                a = fmaf(t[g][1].x, q1.x, a);
                a = fmaf(t[g][1].y, q1.y, a);
                a = fmaf(t[g][2].x, q2.x, a);
                a = fmaf(t[g][2].y, q2.y, a);
                a = fmaf(t[g][3].x, q3.x, a);
                a = fmaf(t[g][3].y, q3.y, a);
                acc[j] = a;
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < RPB; ++j) {
        float a = acc[j];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) red[j][warp] = a;
    }
    __syncthreads();
    if (threadIdx.x < RPB && r0 + (int)threadIdx.x < nrot) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
        scores[r0 + threadIdx.x] = t;
    }
}

// Source voxel of every (rotation, destination voxel) of a small grid, as
// int16 (-1: none): the rotation grid is fixed, so the gather geometry is
// computed once and then streamed from HBM (nrot * d^3 * 2 bytes) instead of
// being recomputed for every map pair.
__global__ void k_prop_srcmap(int d, const float *rotmats, int nrot, int16_t *out) {
    __shared__ float F[9];
    const int r = blockIdx.y;
    if (threadIdx.x < 9) F[threadIdx.x] = rotmats[(size_t)r * 9 + threadIdx.x];
    __syncthreads();
    const int n = d * d * d;
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    out[(size_t)r * n + v] = (int16_t)prop_src(F, d, v);
}

// Scores from float16 voxel-major features and a precomputed source map:
// RPB rotations per block, each target voxel's features loaded once for them.
template <int K8, int RPB>
__global__ void __launch_bounds__(256) k_prop_score_map(const uint4 *ET, const uint4 *EQ, int d,
                                                        const int16_t *srcmap, int nrot, float *scores) {
    __shared__ float red[RPB][32];
    const int r0 = blockIdx.x * RPB;
    const int n = d * d * d;
    float acc[RPB];
#pragma unroll
    for (int j = 0; j < RPB; ++j) acc[j] = 0.f;
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        int sj[RPB];
#pragma unroll
        for (int j = 0; j < RPB; ++j) sj[j] = r0 + j < nrot ? (int)__ldg(srcmap + (size_t)(r0 + j) * n + v) : -1;
        float2 t[K8][4];
#pragma unroll
        for (int g = 0; g < K8; ++g) {
            const uint4 a = __ldg(ET + (size_t)v * K8 + g);
            t[g][0] = __half22float2(*(const __half2 *)&a.x);
            t[g][1] = __half22float2(*(const __half2 *)&a.y);
            t[g][2] = __half22float2(*(const __half2 *)&a.z);
            t[g][3] = __half22float2(*(const __half2 *)&a.w);
        }
#pragma unroll
        for (int j = 0; j < RPB; ++j) {
            const int s = sj[j];
            if (s < 0) continue;
#pragma unroll
            for (int g = 0; g < K8; ++g) {
                const uint4 b = __ldg(EQ + (size_t)s * K8 + g);
                const float2 q0 = __half22float2(*(const __half2 *)&b.x), q1 = __half22float2(*(const __half2 *)&b.y);
                const float2 q2 = __half22float2(*(const __half2 *)&b.z), q3 = __half22float2(*(const __half2 *)&b.w);
                float a = acc[j];
                a = fmaf(t[g][0].x, q0.x, a);
                a = fmaf(t[g][0].y, q0.y, a);
                a = fmaf(t[g][1].x, q1.x, a);
                a = fmaf(t[g][1].y, q1.y, a);
                a = fmaf(t[g][2].x, q2.x, a);
                a = fmaf(t[g][2].y, q2.y, a);
                a = fmaf(t[g][3].x, q3.x, a);
                a = fmaf(t[g][3].y, q3.y, a);
                acc[j] = a;
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < RPB; ++j) {
        float a = acc[j];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) red[j][warp] = a;
    }
    __syncthreads();
    if (threadIdx.x < RPB && r0 + (int)threadIdx.x < nrot) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
        scores[r0 + threadIdx.x] = t;
    }
}

// The same scores with the query's features staged in shared memory: block
// (pair p, chunk c) scores rotations [c kScChunk, (c + 1) kScChunk) of pair p,
// so each rotation's gathers are shared-memory loads instead of scattered L1
// lines, and the blocks of one chunk (consecutive in launch order, pair index
// fastest) read that chunk of the gather map while it is in L2.  Row n of the
// staged features is zero and stands for "no source voxel" (the product of a
// finite feature with +0 adds nothing).  Thread t sums voxels t, t + 256, ...
// in the order of k_prop_score_map and the reduction is the same, so the scores
// are bit-identical to it.  Pair p reads ET + p pstride and EQ + p pstride
// (uint4 units) and writes scores + p nrot.
constexpr int kScChunk = 32;
constexpr int kScRPB = 8;

// c + a.lo * b.lo, then + a.hi * b.hi, for packed float16 pairs a, b: each step
// one fma.rn.f32.f16 (float16 operands, float32 addend and result, one
// rounding), which equals fmaf on the operands converted to float32 (the
// conversion is exact and the product of two float16 values is exact in
// float32).
__device__ __forceinline__ float fma_h2_f32(uint32_t a, uint32_t b, float c) {
    float d;
    asm("{\n\t.reg .f16 al, ah, bl, bh;\n\t"
        "mov.b32 {al, ah}, %1;\n\t"
        "mov.b32 {bl, bh}, %2;\n\t"
        "fma.rn.f32.f16 %0, al, bl, %3;\n\t"
        "fma.rn.f32.f16 %0, ah, bh, %0;\n\t}"
        : "=f"(d) : "r"(a), "r"(b), "f"(c));
    return d;
}
template <int K8>
__global__ void __launch_bounds__(256) k_prop_score_map_s(const uint4 *ET, const uint4 *EQ, size_t pstride,
                                                          int npair, int d, const int16_t *srcmap, int nrot,
                                                          float *scores) {
    extern __shared__ uint4 sq[];   // [n + 1][K8]
    __shared__ float red[kScRPB][8];
    const int n = d * d * d;
    const int p = blockIdx.x % npair, c = blockIdx.x / npair;
    const uint4 *et = ET + (size_t)p * pstride, *eq = EQ + (size_t)p * pstride;
    for (int e = threadIdx.x; e < n * K8; e += blockDim.x) sq[e] = __ldg(eq + e);
    if (threadIdx.x < K8) sq[(size_t)n * K8 + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rend = min(nrot, (c + 1) * kScChunk);
    for (int r0 = c * kScChunk; r0 < rend; r0 += kScRPB) {
        float acc[kScRPB];
#pragma unroll
        for (int j = 0; j < kScRPB; ++j) acc[j] = 0.f;
        for (int v = threadIdx.x; v < n; v += blockDim.x) {
            int sj[kScRPB];
#pragma unroll
            for (int j = 0; j < kScRPB; ++j) {
                const int s = r0 + j < rend ? (int)__ldg(srcmap + (size_t)(r0 + j) * n + v) : -1;
                sj[j] = s < 0 ? n : s;
            }
            uint4 t[K8];
#pragma unroll
            for (int g = 0; g < K8; ++g) t[g] = __ldg(et + (size_t)v * K8 + g);
#pragma unroll
            for (int j = 0; j < kScRPB; ++j) {
#pragma unroll
                for (int g = 0; g < K8; ++g) {
                    const uint4 b = sq[(size_t)sj[j] * K8 + g];
                    float a = acc[j];
                    a = fma_h2_f32(t[g].x, b.x, a);
                    a = fma_h2_f32(t[g].y, b.y, a);
                    a = fma_h2_f32(t[g].z, b.z, a);
                    a = fma_h2_f32(t[g].w, b.w, a);
                    acc[j] = a;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kScRPB; ++j) {
            float a = acc[j];
            for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
            if (lane == 0) red[j][warp] = a;
        }
        __syncthreads();
        if (threadIdx.x < kScRPB && r0 + (int)threadIdx.x < rend) {
            float t = 0.f;
            for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
            scores[(size_t)p * nrot + r0 + threadIdx.x] = t;
        }
        __syncthreads();   // red is rewritten by the next group
    }
}

// ---- the same correlation and its gradients for 8 float32 channels -----------------
// One side's features (the gathered ones) sit in shared memory as two planes of
// float4, so a gathered voxel is two 16-byte loads; row n is zero and stands for
// "no source voxel".  Positions are recomputed: the matrices of a group of
// rotations are in shared memory and a voxel's own coordinates stay in registers,
// about 25 instructions, where the general prop_src takes several times that.
constexpr int kS8Threads = 1024;
constexpr int kS8Rot = 8;      // rotations of a block of k_prop_sources

// Planes [2][n + 1] float4 of channel-major features.
__device__ __forceinline__ void stage_planes(const float *E, int n, float4 *pl) {
    for (int v = threadIdx.x; v < n; v += blockDim.x) {
        pl[v] = make_float4(__ldg(E + v), __ldg(E + n + v), __ldg(E + 2 * n + v), __ldg(E + 3 * n + v));
        pl[n + 1 + v] =
            make_float4(__ldg(E + 4 * n + v), __ldg(E + 5 * n + v), __ldg(E + 6 * n + v), __ldg(E + 7 * n + v));
    }
    if (threadIdx.x == 0) pl[n] = pl[2 * n + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// prop_src with the voxel's first candidate rows (hx, hy, hz: minus the centre)
// at hand; the other candidates of an odd side's middle index are looked at only
// where the first is off the grid, in gather_src's order (z slowest, x, y).
struct Voxel {
    float hx, hy, hz;
    int v;     // destination voxel
    int mid;   // -1: no row; else a bit for each axis with a second row (4 z, 2 x, 1 y)
};
__device__ __forceinline__ Voxel voxel_at(int x, int y, int z, int d) {
    Voxel o;
    o.v = (x * d + y) * d + z;
    o.mid = 0;
    if (d & 1) {
        const int m = (d - 1) >> 1;
        o.mid = d > 1 && (x == d - 1 || y == d - 1 || z == d - 1) ? -1 : (z == m) << 2 | (x == m) << 1 | (y == m);
        x += x >= m;
        y += y >= m;
        z += z >= m;
    }
    const float hc = 0.5f * (float)d;
    o.hx = (float)x - hc;
    o.hy = (float)y - hc;
    o.hz = (float)z - hc;
    return o;
}
__device__ __forceinline__ Voxel voxel_of(int v, int d) { return voxel_at(v / (d * d), v / d % d, v % d, d); }
// A staged matrix (3 float4 of shared memory) in registers.
__device__ __forceinline__ void load_matrix(const float4 *m, float (&F)[9]) {
    const float4 a = m[0], b = m[1], c = m[2];
    F[0] = a.x, F[1] = a.y, F[2] = a.z, F[3] = a.w, F[4] = b.x, F[5] = b.y, F[6] = b.z, F[7] = b.w, F[8] = c.x;
}
__device__ __forceinline__ int voxel_src(const float (&F)[9], int d, const Voxel &o) {
    if (o.mid < 0) return -1;
    const float hc = 0.5f * (float)d;
    int ox, oy, oz;
    if (old_index(F, d, hc, o.hx, o.hy, o.hz, ox, oy, oz)) return (ox * d + oy) * d + oz;
#pragma unroll 1
    for (int k = -o.mid & o.mid; k; k = (k - o.mid) & o.mid)   // the masks within mid, ascending
        if (old_index(F, d, hc, o.hx - (float)(k >> 1 & 1), o.hy - (float)(k & 1), o.hz - (float)(k >> 2), ox, oy, oz))
            return (ox * d + oy) * d + oz;
    return -1;
}

__device__ __forceinline__ float dot8(float4 a0, float4 a1, float4 b0, float4 b1, float s) {
    s = fmaf(a0.x, b0.x, s);
    s = fmaf(a0.y, b0.y, s);
    s = fmaf(a0.z, b0.z, s);
    s = fmaf(a0.w, b0.w, s);
    s = fmaf(a1.x, b1.x, s);
    s = fmaf(a1.y, b1.y, s);
    s = fmaf(a1.z, b1.z, s);
    return fmaf(a1.w, b1.w, s);
}
__device__ __forceinline__ void axpy8(float g, float4 b0, float4 b1, float *acc) {
    acc[0] = fmaf(g, b0.x, acc[0]);
    acc[1] = fmaf(g, b0.y, acc[1]);
    acc[2] = fmaf(g, b0.z, acc[2]);
    acc[3] = fmaf(g, b0.w, acc[3]);
    acc[4] = fmaf(g, b1.x, acc[4]);
    acc[5] = fmaf(g, b1.y, acc[5]);
    acc[6] = fmaf(g, b1.z, acc[6]);
    acc[7] = fmaf(g, b1.w, acc[7]);
}

// scores of rotations [b chunk, (b + 1) chunk): the query's features staged once per
// block.  Each of the block's four groups of 256 threads takes RG rotations at a time,
// so a target voxel's features and coordinates serve RG rotations.  The sums
// are those of k_prop_score, term for term: the gradient of the softmax over the scores
// is a difference of nearly equal numbers, and what a score is off by is what it is off
// by.  Bound by the shared-memory wavefronts of the two gathers per (rotation, voxel).
// Side 15, 24,624 rotations: 656 us with k_prop_score, 254 with RG = 4, 297 with 2;
// 1,008 rotations: 39, 27 and 19 (more blocks).
constexpr int kScSum = 256, kScGroups = kS8Threads / kScSum;
template <int RG>
__global__ void __launch_bounds__(kS8Threads) k_prop_score8(const float *ET, const float *EQ, int d,
                                                            const float *rotmats, int nrot, int chunk, float *scores,
                                                            unsigned md) {
    extern __shared__ float4 pl[];   // [2][n + 1]
    constexpr int kAll = RG * kScGroups;
    __shared__ float4 Fs[kAll][3];
    __shared__ float red[kAll][kScSum / 32];
    const int n = d * d * d, group = threadIdx.x / kScSum, t = threadIdx.x % kScSum;
    stage_planes(EQ, n, pl);
    const int r1 = min(nrot, (int)(blockIdx.x + 1) * chunk);
    for (int r0 = blockIdx.x * chunk; r0 < r1; r0 += kAll) {
        __syncthreads();
        if (threadIdx.x < 9 * kAll) {
            const int j = threadIdx.x / 9, e = threadIdx.x % 9;
            ((float *)Fs[j])[e] = r0 + j < r1 ? rotmats[(size_t)(r0 + j) * 9 + e] : 0.f;
        }
        __syncthreads();
        float acc[RG];
#pragma unroll
        for (int j = 0; j < RG; ++j) acc[j] = 0.f;
        for (int v = t; v < n; v += kScSum) {
            const int q = quot(v, d, md), x = quot(q, d, md);
            const Voxel o = voxel_at(x, q - x * d, v - q * d, d);
            const float4 t0 = make_float4(__ldg(ET + v), __ldg(ET + n + v), __ldg(ET + 2 * n + v), __ldg(ET + 3 * n + v));
            const float4 t1 =
                make_float4(__ldg(ET + 4 * n + v), __ldg(ET + 5 * n + v), __ldg(ET + 6 * n + v), __ldg(ET + 7 * n + v));
#pragma unroll
            for (int j = 0; j < RG; ++j) {
                float F[9];
                load_matrix(Fs[group * RG + j], F);
                const int s = voxel_src(F, d, o);
                const float4 *f = pl + (s < 0 ? n : s);
                const float a = dot8(t0, t1, f[0], f[n + 1], acc[j]);
                acc[j] = s < 0 ? acc[j] : a;
            }
        }
#pragma unroll
        for (int j = 0; j < RG; ++j) {
            float a = acc[j];
            for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
            if ((t & 31) == 0) red[group * RG + j][t >> 5] = a;
        }
        __syncthreads();
        if (threadIdx.x < kAll && r0 + (int)threadIdx.x < r1) {
            float a = 0.f;
            for (int w = 0; w < kScSum / 32; ++w) a += red[threadIdx.x][w];
            scores[r0 + threadIdx.x] = a;
        }
    }
}

// The source voxel of every (rotation, voxel) of a group of rotations, int16
// [rotations][ns] (-1: none; ns = n rounded up to 8).  An odd side's middle voxels,
// whose other candidate rows take a loop, are done apart from the rest so that
// they do not hold up whole warps.
constexpr int kSrcThreads = 512;
__global__ void __launch_bounds__(kSrcThreads) k_prop_sources(int d, int ns, const float *rotmats, int nrot,
                                                             int16_t *table) {
    __shared__ float4 Fs[kS8Rot][3];
    const int r0 = blockIdx.x * kS8Rot, rn = min(kS8Rot, nrot - r0), dd = d * d;
    if (threadIdx.x < 9 * rn)
        ((float *)Fs[threadIdx.x / 9])[threadIdx.x % 9] = rotmats[(size_t)r0 * 9 + threadIdx.x];
    __syncthreads();
    int16_t *out = table + (size_t)r0 * ns;
    auto row = [&](const Voxel &o) {
        for (int j = 0; j < rn; ++j) {
            float F[9];
            load_matrix(Fs[j], F);
            out[(size_t)j * ns + o.v] = (int16_t)voxel_src(F, d, o);
        }
    };
    const int m = (d - 1) >> 1;
    const bool odd = d & 1;
    for (int v = threadIdx.x; v < d * dd; v += kSrcThreads) {
        const Voxel o = voxel_of(v, d);
        if (o.mid <= 0) row(o);
    }
    if (!odd) return;
    const int e1 = dd, e2 = e1 + (d - 1) * d, e3 = e2 + (d - 1) * (d - 1);
    for (int e = threadIdx.x; e < e3; e += kSrcThreads) {   // x = m; else y = m; else z = m
        int x = m, y = e / d, z = e % d;
        if (e >= e2) {
            x = (e - e2) / (d - 1);
            y = (e - e2) % (d - 1);
            x += x >= m;
            y += y >= m;
            z = m;
        } else if (e >= e1) {
            x = (e - e1) / d;
            x += x >= m;
            y = m;
            z = (e - e1) % d;
        }
        row(voxel_at(x, y, z, d));
    }
}

// Target side of the gradient, part[c][0][k][v] (+)= sum over the chunk c of
// rotations of g_r EQ[k][src_r(v)]: a thread owns kT8Own voxels and keeps their 8
// sums in registers (block (p, c): voxels [p, p + 1) kT8Own kS8Threads, chunk c).
// add: the sums go on from the last group of rotations.
constexpr int kT8Own = 4;
__global__ void __launch_bounds__(kS8Threads) k_prop_bwd_t8(const float *EQ, int d, int ns, const int16_t *table,
                                                            int nrot, const float *gs, int chunk, int add,
                                                            float *part) {
    extern __shared__ float4 pl[];   // [2][n + 1]
    const int n = d * d * d;
    stage_planes(EQ, n, pl);
    __syncthreads();
    float acc[kT8Own][8];
#pragma unroll
    for (int i = 0; i < kT8Own; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[i][k] = 0.f;
    const int r1 = min(nrot, (int)(blockIdx.y + 1) * chunk), v0 = blockIdx.x * kT8Own * kS8Threads + threadIdx.x;
#pragma unroll 2
    for (int r = blockIdx.y * chunk; r < r1; ++r) {
        const float g = __ldg(gs + r);
#pragma unroll
        for (int i = 0; i < kT8Own; ++i) {
            const int v = v0 + i * kS8Threads;
            const int s = v < n ? (int)__ldg(table + (size_t)r * ns + v) : -1;
            const float4 *q = pl + (s < 0 || g == 0.f ? n : s);
            axpy8(s < 0 ? 0.f : g, q[0], q[n + 1], acc[i]);
        }
    }
    float *dst = part + (size_t)blockIdx.y * 16 * n;
#pragma unroll
    for (int i = 0; i < kT8Own; ++i) {
        const int v = v0 + i * kS8Threads;
        if (v < n)
#pragma unroll
            for (int k = 0; k < 8; ++k) dst[(size_t)k * n + v] = acc[i][k] + (add ? dst[(size_t)k * n + v] : 0.f);
    }
}

// Query side, part[c][1][k][s] (+)= sum over the chunk's rotations of g_r sum of
// ET[k][v] over the v with src_r(v) = s.  Scattering the 8 channels with
// shared-memory float atomics (compare-and-swap loops) took most of the backward
// pass; instead each rotation's voxels are linked into a list per source (one
// integer exchange each), and a thread owns kS8Own sources, follows their lists and
// keeps the sums in registers.  NB rotations between two barriers, as many as shared
// memory holds lists for.
// Measured at side 15, 24,624 rotations: both sides together 6.12 ms with atomics; now
// source table 0.23, target side 0.29, query side 0.48, the last two bound by the
// shared-memory wavefronts of their gathers.
constexpr int kS8Own = 4;
template <int NB>
__global__ void __launch_bounds__(kS8Threads) k_prop_bwd_q8(const float *ET, int d, int ns, const int16_t *table,
                                                            int nrot, const float *gs, int chunk, int add,
                                                            float *part) {
    extern __shared__ float4 pl[];   // [2][n + 1], then int head[NB][kOwned], int16 next[NB][ns]
    constexpr int kOwned = kS8Own * kS8Threads;
    const int n = d * d * d, s0 = blockIdx.x * kOwned;
    int *head = (int *)(pl + 2 * (n + 1));
    int16_t *next = (int16_t *)(head + NB * kOwned);
    stage_planes(ET, n, pl);
    for (int e = threadIdx.x; e < NB * kOwned; e += kS8Threads) head[e] = -1;
    float acc[kS8Own][8];
#pragma unroll
    for (int i = 0; i < kS8Own; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[i][k] = 0.f;
    const int r1 = min(nrot, (int)(blockIdx.y + 1) * chunk);
    for (int r = blockIdx.y * chunk; r < r1; r += NB) {
        __syncthreads();
        for (int v = threadIdx.x; v < n; v += kS8Threads) {
            unsigned s[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b)   // -1 - s0 wraps past kOwned
                s[b] = r + b < r1 ? (unsigned)((int)__ldg(table + (size_t)(r + b) * ns + v) - s0) : ~0u;
#pragma unroll
            for (int b = 0; b < NB; ++b)
                if (s[b] < (unsigned)kOwned) next[b * ns + v] = (int16_t)atomicExch(head + b * kOwned + s[b], v);
        }
        __syncthreads();
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const float g = r + b < r1 ? __ldg(gs + r + b) : 0.f;
#pragma unroll
            for (int i = 0; i < kS8Own; ++i) {
                int *h = head + b * kOwned + i * kS8Threads + threadIdx.x;
                int v = *h;
                *h = -1;
                if (g == 0.f) continue;
                while (v >= 0) {
                    axpy8(g, pl[v], pl[n + 1 + v], acc[i]);
                    v = next[b * ns + v];
                }
            }
        }
    }
    float *dst = part + (size_t)blockIdx.y * 16 * n + (size_t)8 * n;
#pragma unroll
    for (int i = 0; i < kS8Own; ++i) {
        const int s = s0 + i * kS8Threads + threadIdx.x;
        if (s < n)
#pragma unroll
            for (int k = 0; k < 8; ++k) dst[(size_t)k * n + s] = acc[i][k] + (add ? dst[(size_t)k * n + s] : 0.f);
    }
}

// Partial gradients of the correlation for channels [k0, k0 + kc): block b
// takes rotations [b*chunk, (b+1)*chunk) and writes part[b][0][k][v] =
// sum_r g_r EQ[k][src_r(v)] and part[b][1][k][s] = sum_r g_r ET[k][v] summed
// over the v with src_r(v) = s, accumulated in shared memory.
__global__ void k_prop_score_bwd(const float *ET, const float *EQ, int K, int k0, int kc, int d,
                                 const float *rotmats, int nrot, const float *gs, int chunk, float *part) {
    extern __shared__ __align__(16) float sm[];
    const int n = d * d * d;
    float *gT = sm;             // [kc][n]
    float *gQ = sm + kc * n;    // [kc][n]
    __shared__ float F[9];
    for (int i = threadIdx.x; i < 2 * kc * n; i += blockDim.x) sm[i] = 0.f;
    const int r0 = blockIdx.x * chunk, r1 = min(nrot, r0 + chunk);
    for (int r = r0; r < r1; ++r) {
        __syncthreads();
        if (threadIdx.x < 9) F[threadIdx.x] = rotmats[(size_t)r * 9 + threadIdx.x];
        __syncthreads();
        const float g = gs[r];
        if (g == 0.f) continue;
        for (int v = threadIdx.x; v < n; v += blockDim.x) {
            const int s = prop_src(F, d, v);
            if (s < 0) continue;
            for (int k = 0; k < kc; ++k) {
                gT[k * n + v] = fmaf(g, EQ[(size_t)(k0 + k) * n + s], gT[k * n + v]);
                atomicAdd(&gQ[k * n + s], g * ET[(size_t)(k0 + k) * n + v]);
            }
        }
    }
    __syncthreads();
    float *dst = part + (size_t)blockIdx.x * 2 * K * n;
    for (int i = threadIdx.x; i < 2 * kc * n; i += blockDim.x) {
        const int half = i / (kc * n), rem = i % (kc * n);
        dst[(size_t)half * K * n + (size_t)k0 * n + rem] = sm[i];
    }
}

__global__ void k_sum_parts(const float *part, int nparts, int len, float *out_a, float *out_b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * len) return;
    float s = 0.f;
    for (int p = 0; p < nparts; ++p) s += part[(size_t)p * 2 * len + i];
    if (i < len)
        out_a[i] += s;
    else
        out_b[i - len] += s;
}

// ---- loss ---------------------------------------------------------------------
// Block-wide sum / max of one value per thread (blockDim a multiple of 32).
__device__ float block_sum(float v, float *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < nw; ++w) t += red[w];
    return t;
}
__device__ float block_max(float v, float *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float t = -INFINITY;
    for (int w = 0; w < nw; ++w) t = fmaxf(t, red[w]);
    return t;
}

// Standardised scores u = (s - mean) / std over the rotations, p =
// softmax(u / tau), loss += -sum q log p, and the gradient with respect to s
// through the standardisation:
//   gu = (p - q) / tau,  gs = (gu - mean(gu) - u * mean(gu * u)) / std.
// One block; three passes over the n scores.
__global__ void k_softmax_ce(const float *s, const float *q, int n, float tau, float *loss, float *g) {
    __shared__ float red[32];
    float a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += s[i];
    const float mu = block_sum(a, red) / (float)n;
    a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float t = s[i] - mu;
        a = fmaf(t, t, a);
    }
    const float sd = sqrtf(block_sum(a, red) / (float)n) + 1e-6f;
    const float inv = 1.f / sd;
    float m = -INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, (s[i] - mu) * inv / tau);
    m = block_max(m, red);
    a = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += expf((s[i] - mu) * inv / tau - m);
    const float lz = logf(block_sum(a, red));
    float l = 0.f, sg = 0.f, sgu = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float u = (s[i] - mu) * inv;
        const float lp = u / tau - m - lz;
        l -= q[i] * lp;
        const float gu = (expf(lp) - q[i]) / tau;
        g[i] = gu;
        sg += gu;
        sgu = fmaf(gu, u, sgu);
    }
    l = block_sum(l, red);
    const float mg = block_sum(sg, red) / (float)n;
    const float mgu = block_sum(sgu, red) / (float)n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float u = (s[i] - mu) * inv;
        g[i] = (g[i] - mg - u * mgu) * inv;
    }
    if (threadIdx.x == 0) *loss += l;
}

// ---- Adam (float32 master weights, bfloat16 copies for the convolutions) ------
__global__ void k_adam(float *w, float *m, float *v, const float *g, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, float gscale, __nv_bfloat16 *wbf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] * gscale;
    m[i] = b1 * m[i] + (1.f - b1) * gi;
    v[i] = b2 * v[i] + (1.f - b2) * gi * gi;
    w[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
    if (wbf) wbf[i] = __float2bfloat16(w[i]);
}

// ---- top-k subset: indices of the k largest scores (ties to lower index) --------
// One block: the k-th largest order-preserving key by a most-significant-digit
// radix select (four passes of 8 bits over per-warp shared histograms), then
// an ordered compaction.  The keys sit in shared memory when they fit
// (skeys), else they are re-read from global memory each pass.
constexpr int kTkWarps = 1024 / 32;
__global__ void __launch_bounds__(1024) k_topk_subset(const float *s, int n, int k, int32_t *idx, int skeys) {
    extern __shared__ uint32_t dyn[];
    uint32_t *hist = dyn;                       // [kTkWarps][256] per-warp digit counts
    uint32_t *keys = dyn + kTkWarps * 256;      // [n] when skeys
    __shared__ unsigned int cnt;
    __shared__ int ncount[1024 / 32];
    __shared__ uint32_t sel_digit, sel_need;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s += (size_t)blockIdx.x * n;     // block b: score row b
    idx += (size_t)blockIdx.x * k;
    if (skeys) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) keys[i] = float_order(s[i]);
    }
    __syncthreads();
    auto key = [&](int i) -> uint32_t { return skeys ? keys[i] : float_order(s[i]); };
    // digits from the top: prefix/mask select the keys that still compete;
    // need = how many of the k still have to come from them
    uint32_t prefix = 0u, mask = 0u, need = (uint32_t)k;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < kTkWarps * 256; i += blockDim.x) hist[i] = 0u;
        __syncthreads();
        uint32_t *hw = hist + warp * 256;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint32_t kv = key(i);
            if ((kv & mask) == prefix) atomicAdd(&hw[(kv >> shift) & 255u], 1u);
        }
        __syncthreads();
        // fold the warps' histograms into the first one
        for (int b = threadIdx.x; b < 256; b += blockDim.x) {
            uint32_t t = 0;
            for (int w = 0; w < kTkWarps; ++w) t += hist[w * 256 + b];
            hist[b] = t;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t cum = 0, d = 0, nd = need;
            for (int b = 255; b >= 0; --b) {
                const uint32_t c = hist[b];
                if (cum + c >= need) {
                    d = (uint32_t)b;
                    nd = need - cum;
                    break;
                }
                cum += c;
            }
            sel_digit = d;
            sel_need = nd;
        }
        __syncthreads();
        prefix |= sel_digit << shift;
        mask |= 255u << shift;
        need = sel_need;
        __syncthreads();
    }
    const uint32_t t = prefix;   // the k-th largest key: count(key > t) < k <= count(key >= t)
    // strictly above the threshold first, then ties in index order, k in total
    if (threadIdx.x == 0) cnt = 0u;
    __syncthreads();
    unsigned int above = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) above += key(i) > t;
    for (int o = 16; o > 0; o >>= 1) above += __shfl_down_sync(0xffffffffu, above, o);
    if (lane == 0) atomicAdd(&cnt, above);
    __syncthreads();
    const int n_above = (int)cnt;
    // one ordered compaction: every index above the threshold and the first
    // (k - n_above) ties, in ascending index order
    const int ties_wanted = k - n_above;
    int base_sel = 0, base_tie = 0;
    for (int start = 0; start < n; start += blockDim.x) {
        const int i = start + threadIdx.x;
        const uint32_t kv = i < n ? key(i) : 0u;
        const int is_above = i < n && kv > t, is_tie = i < n && kv == t;
        const unsigned lower = (1u << lane) - 1u;
        // tie positions first (warp ballot, then a prefix over the warps)
        const unsigned mt = __ballot_sync(0xffffffffu, is_tie);
        if (lane == 0) ncount[warp] = __popc(mt);
        __syncthreads();
        int pt = 0, tt = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            if (w < warp) pt += ncount[w];
            tt += ncount[w];
        }
        const int sel = is_above || (is_tie && base_tie + pt + __popc(mt & lower) < ties_wanted);
        __syncthreads();
        const unsigned ms = __ballot_sync(0xffffffffu, sel);
        if (lane == 0) ncount[warp] = __popc(ms);
        __syncthreads();
        int ps = 0, ts = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            if (w < warp) ps += ncount[w];
            ts += ncount[w];
        }
        if (sel) idx[base_sel + ps + __popc(ms & lower)] = i;
        base_sel += ts;
        base_tie += tt;
        __syncthreads();
    }
}

}  // namespace vg

using namespace vg;

extern "C" int vesper_prop_field(const double *data, const float *vec, int d, int pool, float *out, void *stream) {
    if (!data || !vec || !out || d < 1 || pool < 1) return fail(VESPER_ERR_INVALID, "prop_field: bad args");
    const int dp = (d + pool - 1) / pool;
    const int np = dp * dp * dp;
    k_prop_field<<<(np + 127) / 128, 128, 0, (cudaStream_t)stream>>>(data, vec, d, pool, dp, out);
    VG_CHECK_LAUNCH("k_prop_field");
    return VESPER_OK;
}

extern "C" int vesper_prop_conv_fwd(const float *in, int cin, const void *W, const float *bias, int cout, int d,
                                    int relu, int nmap, float *out, void *stream) {
    if (!in || !W || !out || cin < 1 || cout < 1 || d < 1 || nmap < 1 || nmap > 65535)
        return fail(VESPER_ERR_INVALID, "conv_fwd: bad args");
    const int n = d * d * d;
    if (conv_s<false>(in, nullptr, (const __nv_bfloat16 *)W, bias, cin, cout, d, relu, nmap, out,
                          (cudaStream_t)stream)) {
        VG_CHECK_LAUNCH("k_conv_s");
        return VESPER_OK;
    }
    k_conv_fwd<<<dim3((n + 127) / 128, cout, nmap), 128, 0, (cudaStream_t)stream>>>(
        in, cin, (const __nv_bfloat16 *)W, bias, cout, d, relu, out);
    VG_CHECK_LAUNCH("k_conv_fwd");
    return VESPER_OK;
}

extern "C" int vesper_prop_conv_bwd(const float *dout, const float *out, int relu, const float *in, const void *W,
                                    int cin, int cout, int d, float *din, float *dW, float *db, void *stream) {
    if (!dout || !out || !in || !W || !dW || !db || cin < 1 || cout < 1 || d < 1)
        return fail(VESPER_ERR_INVALID, "conv_bwd: bad args");
    const int n = d * d * d;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t smw = (size_t)(d + 2) * (d + 2) * (d + 2) * sizeof(float);
    if (din && conv_s<true>(dout, relu ? out : nullptr, (const __nv_bfloat16 *)W, nullptr, cout, cin, d, 0, 1, din,
                                st)) {
        VG_CHECK_LAUNCH("k_conv_s");
    } else if (din) {
        k_conv_bwd_data<<<dim3((n + 127) / 128, cin), 128, 0, st>>>(dout, out, relu, (const __nv_bfloat16 *)W, cin,
                                                                    cout, d, din);
        VG_CHECK_LAUNCH("k_conv_bwd_data");
    }
    if (cout % kWgCo == 0 && smw + 8192 <= (size_t)smem_limit()) {
        allow_smem(k_conv_bwd_weight_s, smw);
        k_conv_bwd_weight_s<<<cout / kWgCo * cin, kWgThreads, smw, st>>>(dout, out, relu, in, cin, cout, d, dW, db, recip(d),
                                                                         recip(d + 2));
        VG_CHECK_LAUNCH("k_conv_bwd_weight_s");
        return VESPER_OK;
    }
    k_conv_bwd_weight<<<cout * cin, 256, 0, st>>>(dout, out, relu, in, cin, cout, d, dW, db);
    VG_CHECK_LAUNCH("k_conv_bwd_weight");
    return VESPER_OK;
}

// Shared memory of the 8-channel kernels (two planes of features; the query side of
// the gradient also keeps its lists), or 0 where it does not fit (sides above 18;
// those take the general kernels).
static size_t score8_smem(int d, int lists) {
    if (d > 31) return 0;   // int16 voxel indices
    const size_t n = (size_t)d * d * d;
    const size_t b = 2 * (n + 1) * sizeof(float4) +
                     lists * (kS8Own * kS8Threads * sizeof(int) + ((n + 7) & ~(size_t)7) * sizeof(int16_t));
    return b + 4096 <= (size_t)smem_limit() ? b : 0;
}
// Rotations per block: whole groups of `whole`, about `blocks` blocks in all.
static int score8_chunk(int nrot, int blocks, int whole) {
    const int per = (nrot + blocks - 1) / blocks;
    return (per + whole - 1) / whole * whole;
}
template <int RG>
static void score8(const float *ET, const float *EQ, int d, const float *rotmats, int nrot, size_t sm, float *scores,
                   cudaStream_t st) {
    const int chunk = score8_chunk(nrot, kPropSMs, RG * kScGroups);
    allow_smem(k_prop_score8<RG>, sm);
    k_prop_score8<RG><<<(nrot + chunk - 1) / chunk, kS8Threads, sm, st>>>(ET, EQ, d, rotmats, nrot, chunk, scores,
                                                                          recip(d));
}

extern "C" int vesper_prop_score(const float *ET, const float *EQ, int K, int d, const float *rotmats, int nrot,
                                 float *scores, void *stream) {
    if (!ET || !EQ || !rotmats || !scores || K < 1 || d < 1 || nrot < 0)
        return fail(VESPER_ERR_INVALID, "prop_score: bad args");
    if (nrot == 0) return VESPER_OK;
    // Fewer rotations than three blocks of the general kernel to an SM take one wave
    // there (side 18, 304 rotations: 20.6 us, 26.8 staged; side 12 9.4 and 12.5); from
    // 500 on the staged kernel is the faster one at most sides (18 29.0 and 26.9, 15
    // 22.6 and 18.6, 12 10.4 and 14.4, at 800 16.1 and 14.1).
    const size_t sm8 = nrot < 3 * kPropSMs ? 0 : score8_smem(d, 0);
    if (K == 8 && sm8) {
        // 4 rotations per thread once that leaves every SM a group of 16
        (nrot < 16 * kPropSMs ? score8<2> : score8<4>)(ET, EQ, d, rotmats, nrot, sm8, scores, (cudaStream_t)stream);
        VG_CHECK_LAUNCH("k_prop_score8");
        return VESPER_OK;
    }
    k_prop_score<<<nrot, 256, 0, (cudaStream_t)stream>>>(ET, EQ, K, d, rotmats, nrot, scores);
    VG_CHECK_LAUNCH("k_prop_score");
    return VESPER_OK;
}

extern "C" int vesper_prop_vmajor(const float *in, int K, int d, int nmap, float *out, void *stream) {
    if (!in || !out || K < 1 || d < 1 || nmap < 1 || nmap > 65535) return fail(VESPER_ERR_INVALID, "vmajor: bad args");
    const size_t per = (size_t)K * d * d * d;
    k_vmajor<<<dim3((unsigned)((per + 255) / 256), nmap), 256, 0, (cudaStream_t)stream>>>(in, K, d * d * d, out);
    VG_CHECK_LAUNCH("k_vmajor");
    return VESPER_OK;
}

extern "C" int vesper_prop_score_vm(const float *ET, const float *EQ, int K, int d, const float *rotmats, int nrot,
                                    float *scores, void *stream) {
    if (!ET || !EQ || !rotmats || !scores || d < 1 || nrot < 0 || K < 4 || K % 4 || K > 32)
        return fail(VESPER_ERR_INVALID, "prop_score_vm: bad args (K a multiple of 4, <= 32)");
    if (((uintptr_t)ET | (uintptr_t)EQ) & 15) return fail(VESPER_ERR_INVALID, "prop_score_vm: 16-byte alignment");
    if (nrot == 0) return VESPER_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const float4 *a = (const float4 *)ET, *b = (const float4 *)EQ;
    switch (K / 4) {
        case 1: k_prop_score_vm<1><<<nrot, 256, 0, st>>>(a, b, d, rotmats, scores); break;
        case 2: k_prop_score_vm<2><<<nrot, 256, 0, st>>>(a, b, d, rotmats, scores); break;
        case 4: k_prop_score_vm<4><<<nrot, 256, 0, st>>>(a, b, d, rotmats, scores); break;
        case 8: k_prop_score_vm<8><<<nrot, 256, 0, st>>>(a, b, d, rotmats, scores); break;
        default: return fail(VESPER_ERR_UNSUPPORTED, "prop_score_vm: K = %d", K);
    }
    VG_CHECK_LAUNCH("k_prop_score_vm");
    return VESPER_OK;
}

extern "C" int vesper_prop_vmajor_f16(const float *in, int K, int d, int nmap, void *out, void *stream) {
    if (!in || !out || K < 1 || d < 1 || nmap < 1 || nmap > 65535)
        return fail(VESPER_ERR_INVALID, "vmajor_f16: bad args");
    const size_t per = (size_t)K * d * d * d;
    k_vmajor_f16<<<dim3((unsigned)((per + 255) / 256), nmap), 256, 0, (cudaStream_t)stream>>>(in, K, d * d * d,
                                                                                              (__half *)out);
    VG_CHECK_LAUNCH("k_vmajor_f16");
    return VESPER_OK;
}

extern "C" int vesper_prop_score_f16(const void *ET, const void *EQ, int K, int d, const float *rotmats, int nrot,
                                     float *scores, void *stream) {
    if (!ET || !EQ || !rotmats || !scores || d < 1 || nrot < 0 || K < 8 || K % 8 || K > 32)
        return fail(VESPER_ERR_INVALID, "prop_score_f16: bad args (K a multiple of 8, <= 32)");
    if (((uintptr_t)ET | (uintptr_t)EQ) & 15) return fail(VESPER_ERR_INVALID, "prop_score_f16: 16-byte alignment");
    if (nrot == 0) return VESPER_OK;
    cudaStream_t st = (cudaStream_t)stream;
    constexpr int RPB = 4;
    const unsigned nb = (unsigned)((nrot + RPB - 1) / RPB);
    const uint4 *a = (const uint4 *)ET, *b = (const uint4 *)EQ;
    switch (K / 8) {
        case 1: k_prop_score_f16<1, RPB><<<nb, 256, 0, st>>>(a, b, d, rotmats, nrot, scores); break;
        case 2: k_prop_score_f16<2, RPB><<<nb, 256, 0, st>>>(a, b, d, rotmats, nrot, scores); break;
        case 4: k_prop_score_f16<4, RPB><<<nb, 256, 0, st>>>(a, b, d, rotmats, nrot, scores); break;
        default: return fail(VESPER_ERR_UNSUPPORTED, "prop_score_f16: K = %d", K);
    }
    VG_CHECK_LAUNCH("k_prop_score_f16");
    return VESPER_OK;
}

extern "C" int vesper_prop_srcmap(int d, const float *rotmats, int nrot, void *srcmap_out, void *stream) {
    if (!rotmats || !srcmap_out || d < 1 || nrot < 0 || nrot > 65535)
        return fail(VESPER_ERR_INVALID, "prop_srcmap: bad args");
    if ((long long)d * d * d > 32767) return fail(VESPER_ERR_UNSUPPORTED, "prop_srcmap: d^3 above int16");
    if (nrot == 0) return VESPER_OK;
    const int n = d * d * d;
    k_prop_srcmap<<<dim3((n + 255) / 256, nrot), 256, 0, (cudaStream_t)stream>>>(d, rotmats, nrot,
                                                                                (int16_t *)srcmap_out);
    VG_CHECK_LAUNCH("k_prop_srcmap");
    return VESPER_OK;
}

// launch of k_prop_score_map_s for npair pairs, or false when the query's
// features do not fit in shared memory
static bool score_map_staged(const uint4 *et, const uint4 *eq, size_t pstride, int npair, int K8, int d,
                             const int16_t *m, int nrot, float *scores, cudaStream_t st) {
    const int n = d * d * d;
    const size_t sm = ((size_t)n + 1) * K8 * sizeof(uint4);
    if (sm > (size_t)smem_limit()) return false;
    const unsigned nb = (unsigned)(npair * ((nrot + kScChunk - 1) / kScChunk));
    switch (K8) {
        case 1:
            allow_smem(k_prop_score_map_s<1>, sm);
            k_prop_score_map_s<1><<<nb, 256, sm, st>>>(et, eq, pstride, npair, d, m, nrot, scores);
            return true;
        case 2:
            allow_smem(k_prop_score_map_s<2>, sm);
            k_prop_score_map_s<2><<<nb, 256, sm, st>>>(et, eq, pstride, npair, d, m, nrot, scores);
            return true;
        case 4:
            allow_smem(k_prop_score_map_s<4>, sm);
            k_prop_score_map_s<4><<<nb, 256, sm, st>>>(et, eq, pstride, npair, d, m, nrot, scores);
            return true;
    }
    return false;
}

extern "C" int vesper_prop_score_map(const void *ET, const void *EQ, int K, int d, const void *srcmap, int nrot,
                                     float *scores, void *stream) {
    if (!ET || !EQ || !srcmap || !scores || d < 1 || nrot < 0 || K < 8 || K % 8 || K > 32)
        return fail(VESPER_ERR_INVALID, "prop_score_map: bad args (K a multiple of 8, <= 32)");
    if (((uintptr_t)ET | (uintptr_t)EQ) & 15) return fail(VESPER_ERR_INVALID, "prop_score_map: 16-byte alignment");
    if (nrot == 0) return VESPER_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const uint4 *a = (const uint4 *)ET, *b = (const uint4 *)EQ;
    const int16_t *m = (const int16_t *)srcmap;
    if (score_map_staged(a, b, 0, 1, K / 8, d, m, nrot, scores, st)) {
        VG_CHECK_LAUNCH("k_prop_score_map_s");
        return VESPER_OK;
    }
    constexpr int RPB = 4;
    const unsigned nb = (unsigned)((nrot + RPB - 1) / RPB);
    switch (K / 8) {
        case 1: k_prop_score_map<1, RPB><<<nb, 256, 0, st>>>(a, b, d, m, nrot, scores); break;
        case 2: k_prop_score_map<2, RPB><<<nb, 256, 0, st>>>(a, b, d, m, nrot, scores); break;
        case 4: k_prop_score_map<4, RPB><<<nb, 256, 0, st>>>(a, b, d, m, nrot, scores); break;
        default: return fail(VESPER_ERR_UNSUPPORTED, "prop_score_map: K = %d", K);
    }
    VG_CHECK_LAUNCH("k_prop_score_map");
    return VESPER_OK;
}

extern "C" int vesper_prop_score_map_many(const void *VM, int npair, int K, int d, const void *srcmap, int nrot,
                                          float *scores, void *stream) {
    if (!VM || !srcmap || !scores || npair < 0 || d < 1 || nrot < 0 || K < 8 || K % 8 || K > 32)
        return fail(VESPER_ERR_INVALID, "prop_score_map_many: bad args (K a multiple of 8, <= 32)");
    if ((uintptr_t)VM & 15) return fail(VESPER_ERR_INVALID, "prop_score_map_many: 16-byte alignment");
    if (npair == 0 || nrot == 0) return VESPER_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int K8 = K / 8;
    const size_t per = (size_t)d * d * d * K8;   // uint4 per map
    const uint4 *vm = (const uint4 *)VM;
    const int16_t *m = (const int16_t *)srcmap;
    if (score_map_staged(vm, vm + per, 2 * per, npair, K8, d, m, nrot, scores, st)) {
        VG_CHECK_LAUNCH("k_prop_score_map_s");
        return VESPER_OK;
    }
    for (int i = 0; i < npair; ++i) {
        const int rc = vesper_prop_score_map(vm + 2 * i * per, vm + (2 * i + 1) * per, K, d, srcmap, nrot,
                                             scores + (size_t)i * nrot, stream);
        if (rc != VESPER_OK) return rc;
    }
    return VESPER_OK;
}

extern "C" int vesper_prop_score_bwd_workspace(int K, int d, size_t *bytes) {
    if (!bytes) return fail(VESPER_ERR_INVALID, "bytes is NULL");
    *bytes = (size_t)kPropBlocks * 2 * K * d * d * d * sizeof(float);
    return VESPER_OK;
}

extern "C" int vesper_prop_score_bwd(const float *ET, const float *EQ, int K, int d, const float *rotmats, int nrot,
                                     const float *gscores, float *gET, float *gEQ, void *workspace,
                                     size_t workspace_bytes, void *stream) {
    if (!ET || !EQ || !rotmats || !gscores || !gET || !gEQ || K < 1 || d < 1 || nrot < 1)
        return fail(VESPER_ERR_INVALID, "prop_score_bwd: bad args");
    const int n = d * d * d;
    // channels per launch: the largest divisor of K whose two [kc][n] float
    // buffers fit in shared memory
    int kc = K;
    while (kc > 0 && (K % kc != 0 || (size_t)2 * kc * n * sizeof(float) > (size_t)smem_limit())) --kc;
    if (kc < 1) return fail(VESPER_ERR_UNSUPPORTED, "prop_score_bwd: d^3 too large for shared memory");
    const size_t sm = (size_t)2 * kc * n * sizeof(float);
    const int nblk = std::min(kPropBlocks, nrot);
    const int chunk = (nrot + nblk - 1) / nblk;
    size_t need = 0;
    vesper_prop_score_bwd_workspace(K, d, &need);
    if (!workspace || workspace_bytes < need) return fail(VESPER_ERR_WORKSPACE, "prop_score_bwd: workspace");
    cudaStream_t st = (cudaStream_t)stream;
    // Below side 9 few voxels share a rotation's staging and lists, and few of a block's
    // threads own one: the general kernel up to side 6 (side 6, 24,624 rotations: 180
    // us, 264 staged), at 7 and 8 for few rotations (side 7 24.9 and 28.8 at 304, 37.2
    // and 34.9 at 1,008; side 8 20.8 and 22.9 at 152, 27.2 and 24.9 at 304).
    const bool few = d <= 6 || (d <= 8 && nrot < (d == 7 ? 5 : 2) * kPropSMs);
    const size_t sm8t = few ? 0 : score8_smem(d, 0), sm8q = score8_smem(d, 1);
    if (K == 8 && sm8t && sm8q) {
        // slots of the partial gradients (one per chunk of rotations), then the source
        // table of as many rotations as the workspace holds: groups of equal size
        const int parts = (n + kS8Own * kS8Threads - 1) / (kS8Own * kS8Threads);
        const int slots = std::min(nrot, std::max(1, kPropSMs / parts)), ns = (n + 7) & ~7;
        const size_t used = ((size_t)slots * 16 * n * sizeof(float) + 255) & ~(size_t)255;
        const int fit = (int)std::min<size_t>((need - used) / (ns * sizeof(int16_t)), (size_t)nrot);
        const int groups = (nrot + fit - 1) / fit, per_group = (nrot + groups - 1) / groups;
        int16_t *table = (int16_t *)((char *)workspace + used);
        allow_smem(k_prop_bwd_t8, sm8t);
        const size_t sm4 = score8_smem(d, 4), sm2 = score8_smem(d, 2);
        auto q8 = sm4 ? k_prop_bwd_q8<4> : sm2 ? k_prop_bwd_q8<2> : k_prop_bwd_q8<1>;
        const size_t smq = sm4 ? sm4 : sm2 ? sm2 : sm8q;
        allow_smem(q8, smq);
        for (int r0 = 0; r0 < nrot; r0 += per_group) {
            const int rn = std::min(per_group, nrot - r0), chunk = (per_group + slots - 1) / slots;
            k_prop_sources<<<(rn + kS8Rot - 1) / kS8Rot, kSrcThreads, 0, st>>>(d, ns, rotmats + (size_t)r0 * 9, rn, table);
            VG_CHECK_LAUNCH("k_prop_sources");
            k_prop_bwd_t8<<<dim3((n + kT8Own * kS8Threads - 1) / (kT8Own * kS8Threads), slots), kS8Threads, sm8t, st>>>(EQ, d, ns, table, rn, gscores + r0, chunk,
                                                                         r0 > 0, (float *)workspace);
            VG_CHECK_LAUNCH("k_prop_bwd_t8");
            q8<<<dim3(parts, slots), kS8Threads, smq, st>>>(ET, d, ns, table, rn, gscores + r0, chunk, r0 > 0,
                                                            (float *)workspace);
            VG_CHECK_LAUNCH("k_prop_bwd_q8");
        }
        const int nchunk = slots;
        const int len8 = K * n;
        k_sum_parts<<<(2 * len8 + 255) / 256, 256, 0, st>>>((const float *)workspace, nchunk, len8, gET, gEQ);
        VG_CHECK_LAUNCH("k_sum_parts");
        return VESPER_OK;
    }
    allow_smem(k_prop_score_bwd, sm);
    for (int k0 = 0; k0 < K; k0 += kc) {
        k_prop_score_bwd<<<nblk, 256, sm, st>>>(ET, EQ, K, k0, kc, d, rotmats, nrot, gscores, chunk,
                                                (float *)workspace);
        VG_CHECK_LAUNCH("k_prop_score_bwd");
    }
    const int len = K * n;
    k_sum_parts<<<(2 * len + 255) / 256, 256, 0, st>>>((const float *)workspace, nblk, len, gET, gEQ);
    VG_CHECK_LAUNCH("k_sum_parts");
    return VESPER_OK;
}

extern "C" int vesper_prop_softmax_ce(const float *scores, const float *target, int n, float tau, float *loss,
                                      float *gscores, void *stream) {
    if (!scores || !target || !loss || !gscores || n < 1 || !(tau > 0))
        return fail(VESPER_ERR_INVALID, "softmax_ce: bad args");
    k_softmax_ce<<<1, 1024, 0, (cudaStream_t)stream>>>(scores, target, n, tau, loss, gscores);
    VG_CHECK_LAUNCH("k_softmax_ce");
    return VESPER_OK;
}

extern "C" int vesper_prop_adam(float *w, float *m, float *v, const float *g, int n, float lr, float b1, float b2,
                                float eps, int step, float gscale, void *wbf16, void *stream) {
    if (!w || !m || !v || !g || n < 0 || step < 1) return fail(VESPER_ERR_INVALID, "adam: bad args");
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(w, m, v, g, n, lr, b1, b2, eps, c1, c2, gscale,
                                                              (__nv_bfloat16 *)wbf16);
    VG_CHECK_LAUNCH("k_adam");
    return VESPER_OK;
}

extern "C" int vesper_topk_subset_batch(const float *scores, int nbatch, int n, int k, int32_t *idx_out,
                                        void *stream) {
    if (!scores || !idx_out || nbatch < 1 || nbatch > 65535 || n < 1 || k < 1 || k > n)
        return fail(VESPER_ERR_INVALID, "topk_subset: bad args");
    const size_t hb = (size_t)kTkWarps * 256 * sizeof(uint32_t);
    const size_t kb = (size_t)n * sizeof(uint32_t);
    const int skeys = hb + kb <= (size_t)smem_limit() - 4096 ? 1 : 0;
    const size_t sm = hb + (skeys ? kb : 0);
    allow_smem(k_topk_subset, sm);
    k_topk_subset<<<nbatch, 1024, sm, (cudaStream_t)stream>>>(scores, n, k, idx_out, skeys);
    VG_CHECK_LAUNCH("k_topk_subset");
    return VESPER_OK;
}

extern "C" int vesper_topk_subset(const float *scores, int n, int k, int32_t *idx_out, void *stream) {
    return vesper_topk_subset_batch(scores, 1, n, k, idx_out, stream);
}
