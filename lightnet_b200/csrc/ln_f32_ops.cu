// f32 NCHW operators: the F32TensorOpsBackend subset on the detector path
// (lightnet-cuda/src/lib.rs:460).  CUDA-core kernels in binary32 throughout (no
// reduced-precision tensor-core formats): this path exists for trait fidelity, for
// calibration and as the f32 parity target; the throughput path is the 8-bit one.
#include <cooperative_groups.h>

#include "ln_common.h"
#include "ln_conv_f32_plan.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 256;
inline int blocks_for(int64_t n, int per_block = kThreads) { return (int)((n + per_block - 1) / per_block); }

// Convolution as a blocked GEMM: y[f][pixel] = sum over k = (channel, ky, kx) of w[f][k] * x[tap k of pixel].  Each output is one chain of
// fused multiply-adds in k order, the order of runtime/forward_layers.rs:646-695; where tiles are few the k range is split over the
// CTAs of a cluster (blockIdx.z), which add their chains up in order through distributed shared memory: no second pass over the
// output and no second launch.  Taps outside the image enter the sum as zeros, which leaves it as it is while the weights are finite; an
// output that comes out NaN next to the border is summed again without them (conv_f32_taps).
struct ConvF32 {
    const float* x;
    const float* w;
    const float* bias;  // null = none
    float* y;
    int B, C, H, W, F, k, sx, sy, dil, pad, OH, OW, K, act;
};

__device__ __forceinline__ unsigned long long fma2_f32(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Output (image b, filter f, pixel r) tap by tap, those outside the image skipped as in forward_layers.rs:646-695: an infinite or NaN weight
// on such a tap must not reach the output, and a product with a zero would let it.
__device__ __noinline__ float conv_f32_taps(const ConvF32& p, int b, int f, int r) {
    const int iy0 = r / p.OW * p.sy - p.pad, ix0 = r % p.OW * p.sx - p.pad;
    const float* w = p.w + (int64_t)f * p.K;
    float acc = 0.0f;
    for (int c = 0; c < p.C; ++c, w += p.k * p.k) {
        const float* plane = p.x + ((int64_t)b * p.C + c) * p.H * p.W;
        for (int ky = 0; ky < p.k; ++ky) {
            const int iy = iy0 + ky * p.dil;
            if (iy < 0 || iy >= p.H) continue;
            for (int kx = 0; kx < p.k; ++kx) {
                const int ix = ix0 + kx * p.dil;
                if (ix >= 0 && ix < p.W) acc = fmaf(__ldg(plane + (int64_t)iy * p.W + ix), __ldg(w + ky * p.k + kx), acc);
            }
        }
    }
    return acc;
}

// Whether some tap of pixel r lies outside the image.
__device__ __forceinline__ bool conv_f32_border(const ConvF32& p, int r) {
    const int iy0 = r / p.OW * p.sy - p.pad, ix0 = r % p.OW * p.sx - p.pad;
    const int64_t reach = (int64_t)(p.k - 1) * p.dil;
    return iy0 < 0 || ix0 < 0 || iy0 + reach >= p.H || ix0 + reach >= p.W;
}

// The groups of four outputs that a thread of conv_f32_finish found a NaN in (bit = its turn) and left in y as plain sums: NaNs next to the
// border summed again, then bias and activation.  Out of line: inside the loop that hands tiles over it cost 1 % of a forward.
template <int BN, int T>
__device__ __noinline__ void conv_f32_finish_nan(const ConvF32& p, unsigned bad, int m0, int f0, int n0) {
    const int P = p.OH * p.OW, NP = p.B * P;
    for (; bad; bad &= bad - 1u) {
        const int i = (int)threadIdx.x + (__ffs(bad) - 1) * T, f = f0 + m0 + i / (BN / 4), n = n0 + i % (BN / 4) * 4;
        const float bias = p.bias ? __ldg(p.bias + f) : 0.0f;
        for (int j = 0; j < 4 && n + j < NP; ++j) {
            const int b = (n + j) / P, r = n + j - b * P;
            float* y = p.y + ((int64_t)b * p.F + f) * P + r;
            float v = *y;
            if (isnan(v) && conv_f32_border(p, r)) v = conv_f32_taps(p, b, f, r);
            *y = ln_act_f32(p.act, p.bias ? v + bias : v);
        }
    }
}

// Hands the CTA's tile (one per part of a split k range, side by side in distributed shared memory) to y: the parts added up in order,
// bias, activation, 16-byte stores where the planes allow them.  Called by all threads after the tile is written.
template <int BM, int BN, int T>
__device__ __forceinline__ void conv_f32_finish(const ConvF32& p, float (&tile)[BM][BN], int f0, int n0) {
    cg::cluster_group cluster = cg::this_cluster();
    const int P = p.OH * p.OW, NP = p.B * P, parts = (int)gridDim.z, share = BM / parts;
    if (parts > 1) cluster.sync();
    else __syncthreads();
    const bool vec = (P & 3) == 0;  // four consecutive pixels lie in one image then, at a 16-byte boundary
    static_assert(BM * (BN / 4) <= 32 * T, "a bit for every turn of the loop");
    unsigned bad = 0u, turn = 1u;
    for (int i = (int)threadIdx.x; i < share * (BN / 4); i += T, turn <<= 1) {
        const int m = (int)blockIdx.z * share + i / (BN / 4), c = i % (BN / 4) * 4, f = f0 + m, n = n0 + c;
        if (f >= p.F || n >= NP) continue;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int s = 0; s < parts; ++s) {
            const float4 q = *reinterpret_cast<const float4*>(parts > 1 ? cluster.map_shared_rank(&tile[m][c], s) : &tile[m][c]);
            v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
        }
        if (isnan(v[0] + v[1] + v[2] + v[3])) bad |= turn;  // (inf - inf too, which does no harm)
        else {
            const float bias = p.bias ? __ldg(p.bias + f) : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = ln_act_f32(p.act, p.bias ? v[j] + bias : v[j]);
        }
        const int b = n / P;
        if (vec) *reinterpret_cast<float4*>(p.y + ((int64_t)b * p.F + f) * P + (n - b * P)) = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < NP) {
                    const int bj = (n + j) / P;
                    p.y[((int64_t)bj * p.F + f) * P + (n + j - bj * P)] = v[j];
                }
        }
    }
    if (bad) conv_f32_finish_nan<BN, T>(p, bad, (int)blockIdx.z * share, f0, n0);
    if (parts > 1) cluster.sync();  // nobody leaves while its tile is being read
}

// The main kernel: 1x1 without padding (KS = 1) and 3x3 without dilation (KS = 3), k a multiple of 4.  64 filters x BN pixels per CTA.
// What bounds it is the FMA pipe, and next to it the issue slots and the shared-memory port, so
//   - a thread keeps 8 filters x 8 pixels in registers and multiplies two pixels at a time with packed f32x2 FMAs, each of which takes one
//     issue slot for two cycles of the pipe;
//   - both operands go from global to shared memory with cp.async, a slice of 36 (4 channels x 9 taps: the taps are constant
//     offsets from one pointer, valid or not by one bit of a mask computed once) or 32 channels ahead of the multiplication:
//     no registers, no store instructions, and zero fill for what is outside;
//   - weights stay in their own order, [filter][k], copied 16 bytes at a time and read four k at a time; the eight filters of a thread are
//     eight rows apart, which keeps the reads free of bank conflicts.
// (3x3 C256 -> K512 at 38x38: 146 us with operands staged through registers and k decoded per element -- 38 % of the instructions were
// FMAs --, 139 us with weights transposed into shared memory four bytes at a time: the scatter filled the shared-memory port.)
template <int BN, int KS>
struct ConvF32Shared {
    static constexpr int SL = ln_conv_f32_slice(true, KS), WL = SL + 4;
    union {
        struct { float w[2][64][WL]; float x[2][SL][BN]; } op;
        float tile[64][BN];
    };
};

template <int BN, int KS>
__global__ void __launch_bounds__(BN, 512 / BN) conv2d_f32_async_kernel(const __grid_constant__ ConvF32 p) {
    using Shared = ConvF32Shared<BN, KS>;
    constexpr int T = BN, TX = BN / 8, SL = Shared::SL, WCOPIES = (64 * SL / 4 + T - 1) / T;
    extern __shared__ __align__(16) unsigned char smem[];
    Shared& sm = *reinterpret_cast<Shared*>(smem);
    const int tid = (int)threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int P = p.OH * p.OW, HW = p.H * p.W, NP = p.B * P;
    const int n0 = (int)blockIdx.x * BN, f0 = (int)blockIdx.y * 64;
    const int slices = (p.K + SL - 1) / SL, z = (int)blockIdx.z, parts = (int)gridDim.z;
    const int k_begin = ln_conv_f32_first_slice(slices, z, parts) * SL, k_end = min(p.K, ln_conv_f32_first_slice(slices, z + 1, parts) * SL);
    // this thread's pixel: address of tap (0, 0) of the first channel of the range, and the taps inside the image as 4-byte copy sizes
    const int n = n0 + tid;
    const bool real = n < NP;
    const int b = real ? n / P : 0, r = real ? n - b * P : 0, oy = r / p.OW, ox = r - oy * p.OW;
    const int iy0 = oy * p.sy - p.pad, ix0 = ox * p.sx - p.pad;
    const float* px = p.x + ((int64_t)b * p.C + k_begin / (KS * KS)) * HW + (int64_t)iy0 * p.W + ix0;
    unsigned inside = 0u;  // bit t + 2 = tap t
    if (real) {
        if (KS == 1) inside = 4u;
        else
#pragma unroll
            for (int t = 0; t < 9; ++t)
                if (iy0 + t / 3 >= 0 && iy0 + t / 3 < p.H && ix0 + t % 3 >= 0 && ix0 + t % 3 < p.W) inside |= 4u << t;
    }
    // 1x1 stride 1 over planes of a multiple of 4: the tile's pixels are consecutive in memory, four per copy (thread: row tid / (BN / 4))
    const bool x_vec = KS == 1 && p.sx == 1 && p.sy == 1 && (P & 3) == 0 && (((uintptr_t)p.x) & 15) == 0;
    const int vn = n0 + (tid % (BN / 4)) * 4, vb = vn < NP ? vn / P : 0;
    const float* vx = p.x + ((int64_t)vb * p.C + k_begin + tid / (BN / 4)) * HW + (vn < NP ? vn - vb * P : 0);
    const float* wbase = p.w + (int64_t)f0 * p.K;
    auto copy4 = [](const void* dst, const float* src, unsigned bytes) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
    };
    auto copy16 = [](const void* dst, const float* src, unsigned bytes) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
    };
    auto copy_slice = [&](int k0, int buf) {
        const int left = k_end - k0;  // rows of the range from here on; the rest of the slice is filled with zeros
#pragma unroll
        for (int q = 0; q < WCOPIES; ++q) {
            const int i = tid + q * T, m = i / (SL / 4), t = i % (SL / 4) * 4;
            if ((64 * SL / 4) % T != 0 && m >= 64) break;
            const bool ok = f0 + m < p.F && t < left;
            copy16(&sm.op.w[buf][m][t], ok ? wbase + (int64_t)m * p.K + (k0 + t) : p.w, ok ? 16u : 0u);
        }
        if (KS == 3) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool ok = c * 9 < left;
                const float* q0 = ok ? px : p.x;
                const float* q1 = q0 + (ok ? p.W : 0);
                const float* q2 = q1 + (ok ? p.W : 0);
                const unsigned mask = ok ? inside : 0u;
#pragma unroll
                for (int t = 0; t < 9; ++t) copy4(&sm.op.x[buf][c * 9 + t][tid], (mask >> t) & 4u ? (t < 3 ? q0 : (t < 6 ? q1 : q2)) + t % 3 : p.x, (mask >> t) & 4u);
                px += HW;
            }
        } else if (x_vec) {
#pragma unroll
            for (int q = 0; q < SL / 4; ++q) {
                const int row = tid / (BN / 4) + q * 4;
                const bool ok = vn < NP && row < left;
                copy16(&sm.op.x[buf][row][(tid % (BN / 4)) * 4], ok ? vx : p.x, ok ? 16u : 0u);
                vx += (int64_t)4 * HW;
            }
        } else {
#pragma unroll
            for (int c = 0; c < SL; ++c) {
                const bool ok = inside && c < left;
                copy4(&sm.op.x[buf][c][tid], ok ? px : p.x, ok ? 4u : 0u);
                px += HW;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned long long acc[8][4];  // filter ty + 8 i x pixel pairs
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][q] = 0ull;
    copy_slice(k_begin, 0);
    int buf = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += SL) {
        if (k0 + SL < k_end) {
            copy_slice(k0 + SL, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int g = 0; g < SL / 4; ++g) {
            float4 w[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) w[m] = *reinterpret_cast<const float4*>(&sm.op.w[buf][ty + 8 * m][4 * g]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(&sm.op.x[buf][4 * g + e][tx * 4]), xb = *reinterpret_cast<const ulonglong2*>(&sm.op.x[buf][4 * g + e][BN / 2 + tx * 4]);
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const float v = e == 0 ? w[m].x : (e == 1 ? w[m].y : (e == 2 ? w[m].z : w[m].w));
                    unsigned long long w2;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(w2) : "f"(v));
                    acc[m][0] = fma2_f32(w2, xa.x, acc[m][0]);
                    acc[m][1] = fma2_f32(w2, xa.y, acc[m][1]);
                    acc[m][2] = fma2_f32(w2, xb.x, acc[m][2]);
                    acc[m][3] = fma2_f32(w2, xb.y, acc[m][3]);
                }
            }
        }
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        *reinterpret_cast<ulonglong2*>(&sm.tile[ty + 8 * m][tx * 4]) = make_ulonglong2(acc[m][0], acc[m][1]);
        *reinterpret_cast<ulonglong2*>(&sm.tile[ty + 8 * m][BN / 2 + tx * 4]) = make_ulonglong2(acc[m][2], acc[m][3]);
    }
    conv_f32_finish<64, BN, T>(p, sm.tile, f0, n0);
}

// Layers of few filters and every other geometry: BM filters x BN pixels, operands staged through registers (the weights with 4-byte
// copies), slices of one channel for 3x3 kernels (KS = 3) and of eight k otherwise (KS = 1: 1x1 without padding, 0: anything).
template <int BM, int BN, int KS>
__global__ void __launch_bounds__(BM * BN / 64, 32768 / (BM * BN)) conv2d_f32_gemm_kernel(const __grid_constant__ ConvF32 p) {
    constexpr int T = BM * BN / 64, TX = BN / 8, SL = ln_conv_f32_slice(false, KS);
    static_assert(BN % T == 0, "every thread gathers whole columns of x");
    constexpr int PIX = BN / T;                   // pixels a thread gathers
    constexpr int WQ = (BM * SL + T - 1) / T;     // weights a thread copies: element tid + q * T of [filter][k of the slice]
    constexpr int WL = BM + 4;                    // (padded: the copies of a warp scatter over several rows)
    struct Operands { float w[2][SL][WL]; float2 x[2][SL][BN]; };
    __shared__ __align__(16) union { Operands op; float tile[BM][BN]; } sm;
    const int tid = (int)threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int P = p.OH * p.OW, HW = p.H * p.W, NP = p.B * P;
    const int n0 = (int)blockIdx.x * BN, f0 = (int)blockIdx.y * BM;
    const int slices = (p.K + SL - 1) / SL, z = (int)blockIdx.z, parts = (int)gridDim.z;
    const int k_begin = ln_conv_f32_first_slice(slices, z, parts) * SL, k_end = min(p.K, ln_conv_f32_first_slice(slices, z + 1, parts) * SL);
    // the pixels this thread gathers: address of tap (0, 0) of the first channel of the range, and which taps are inside the image
    const float* px[PIX];
    unsigned inside[PIX];
    int oy0[PIX], ox0[PIX];
    const int c_begin = KS == 3 ? k_begin / 9 : (KS == 1 ? k_begin : 0);
#pragma unroll
    for (int j = 0; j < PIX; ++j) {
        const int n = n0 + tid + j * T;
        const bool real = n < NP;
        const int b = n / P, r = n - b * P, oy = r / p.OW, ox = r - oy * p.OW;
        oy0[j] = real ? oy * p.sy - p.pad : 0;
        ox0[j] = ox * p.sx - p.pad;
        px[j] = p.x + ((int64_t)(real ? b : 0) * p.C + c_begin) * HW + (int64_t)oy0[j] * p.W + ox0[j];
        inside[j] = real ? 1u : 0u;  // (KS = 3: a bit per tap instead)
        if (KS == 3) inside[j] = 0u;
        if (KS == 3 && real)
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int iy = oy0[j] + t / 3, ix = ox0[j] + t % 3;
                if (iy >= 0 && iy < p.H && ix >= 0 && ix < p.W) inside[j] |= 1u << t;
            }
    }
    const float* wbase = p.w + (int64_t)f0 * p.K;
    int woff[WQ];  // from wbase, -1: no such filter
#pragma unroll
    for (int q = 0; q < WQ; ++q) {
        const int i = tid + q * T, m = i / SL;
        woff[q] = m < BM && f0 + m < p.F ? m * p.K + (i - m * SL) : -1;
    }
    float gx[SL][PIX];
    auto fetch = [&](int k0) {
        if constexpr (KS == 3) {
#pragma unroll
            for (int j = 0; j < PIX; ++j) {
                const float* q0 = px[j];
                const float* q1 = q0 + p.W;
                const float* q2 = q1 + p.W;
#pragma unroll
                for (int t = 0; t < 9; ++t) gx[t][j] = (inside[j] >> t) & 1u ? __ldg((t < 3 ? q0 : (t < 6 ? q1 : q2)) + t % 3) : 0.0f;
                px[j] += HW;
            }
        } else {
#pragma unroll
            for (int j = 0; j < PIX; ++j) {
                if constexpr (KS == 1) {
                    const float* q = px[j];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        gx[i][j] = inside[j] && k0 + i < k_end ? __ldg(q) : 0.0f;
                        q += HW;
                    }
                    px[j] = q;
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int kr = k0 + i, c = kr / (p.k * p.k), tap = kr - c * p.k * p.k, ky = tap / p.k, kx = tap - ky * p.k;
                        const int iy = oy0[j] + ky * p.dil, ix = ox0[j] + kx * p.dil;
                        const bool ok = inside[j] && kr < k_end && iy >= 0 && iy < p.H && ix >= 0 && ix < p.W;
                        gx[i][j] = ok ? __ldg(px[j] + (int64_t)c * HW + (int64_t)(ky * p.dil) * p.W + kx * p.dil) : 0.0f;
                    }
                }
            }
        }
    };
    auto copy_weights = [&](int k0, int buf) {
#pragma unroll
        for (int q = 0; q < WQ; ++q) {
            const int i = tid + q * T, m = i / SL, t = i - m * SL;
            if ((BM * SL) % T != 0 && m >= BM) break;
            const bool ok = woff[q] >= 0 && (KS == 3 || k0 + t < k_end);
            const float* src = wbase + (ok ? woff[q] + k0 : 0);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(&sm.op.w[buf][t][m])), "l"(src), "r"(ok ? 4 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < SL; ++i)
#pragma unroll
            for (int j = 0; j < PIX; ++j) sm.op.x[buf][i][tid + j * T] = make_float2(gx[i][j], gx[i][j]);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    };
    unsigned long long acc[4][8];  // filters 2i, 2i + 1 of the thread x its eight pixels
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 8; ++n) acc[m][n] = 0ull;
    copy_weights(k_begin, 0);
    fetch(k_begin);
    store(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += SL) {
        const bool more = k0 + SL < k_end;
        if (more) {
            copy_weights(k0 + SL, buf ^ 1);
            fetch(k0 + SL);
        }
#pragma unroll
        for (int r = 0; r < SL; ++r) {
            const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(&sm.op.w[buf][r][ty * 8]), wb = *reinterpret_cast<const ulonglong2*>(&sm.op.w[buf][r][ty * 8 + 4]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // pixels 2 tx + (BN / 4) q and the one after it
                const ulonglong2 x2 = *reinterpret_cast<const ulonglong2*>(&sm.op.x[buf][r][q * (BN / 4) + tx * 2]);
                acc[0][2 * q] = fma2_f32(wa.x, x2.x, acc[0][2 * q]);
                acc[1][2 * q] = fma2_f32(wa.y, x2.x, acc[1][2 * q]);
                acc[2][2 * q] = fma2_f32(wb.x, x2.x, acc[2][2 * q]);
                acc[3][2 * q] = fma2_f32(wb.y, x2.x, acc[3][2 * q]);
                acc[0][2 * q + 1] = fma2_f32(wa.x, x2.y, acc[0][2 * q + 1]);
                acc[1][2 * q + 1] = fma2_f32(wa.y, x2.y, acc[1][2 * q + 1]);
                acc[2][2 * q + 1] = fma2_f32(wb.x, x2.y, acc[2][2 * q + 1]);
                acc[3][2 * q + 1] = fma2_f32(wb.y, x2.y, acc[3][2 * q + 1]);
            }
        }
        if (more) store(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float a0, b0, a1, b1;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(b0) : "l"(acc[m][2 * q]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a1), "=f"(b1) : "l"(acc[m][2 * q + 1]));
            *reinterpret_cast<float2*>(&sm.tile[ty * 8 + 2 * m][q * (BN / 4) + tx * 2]) = make_float2(a0, a1);
            *reinterpret_cast<float2*>(&sm.tile[ty * 8 + 2 * m + 1][q * (BN / 4) + tx * 2]) = make_float2(b0, b1);
        }
    conv_f32_finish<BM, BN, T>(p, sm.tile, f0, n0);
}

// Grouped convolutions, sizes that the blocked kernels do not number (ln_conv_f32_blocked) and those where their tiles are mostly empty
// (ln_conv_f32_per_tap): one thread per (pixel, group of FPT filters).  Semantics of runtime/forward_layers.rs:646-695: taps outside
// the image are skipped, groups partition channels, weights are [filters][C/groups][k][k].
template <int FPT>
__global__ void conv2d_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int B, int C,
                                  int H, int W, int F, int k, int sx, int sy, int dil, int pad, int groups, int OH, int OW) {
    const int fgroups = (F + FPT - 1) / FPT;
    const int64_t total = (int64_t)B * fgroups * OH * OW;
    const int cpg = C / groups, fpg = F / groups;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        int ox = (int)(idx % OW);
        int oy = (int)((idx / OW) % OH);
        int fg = (int)((idx / ((int64_t)OW * OH)) % fgroups);
        int b = (int)(idx / ((int64_t)OW * OH * fgroups));
        float acc[FPT];
#pragma unroll
        for (int j = 0; j < FPT; ++j) acc[j] = 0.0f;
        const int f0 = fg * FPT;
        // all FPT filters share a group only when FPT divides fpg; otherwise fall back to per-filter groups
        const bool same_group = (fpg % FPT) == 0;
        if (same_group) {
            const int g = f0 / fpg;
            for (int ic = 0; ic < cpg; ++ic) {
                const float* xp = x + ((int64_t)b * C + g * cpg + ic) * H * W;
                for (int ky = 0; ky < k; ++ky) {
                    int iy = oy * sy + ky * dil - pad;
                    if (iy < 0 || iy >= H) continue;
                    for (int kx = 0; kx < k; ++kx) {
                        int ix = ox * sx + kx * dil - pad;
                        if (ix < 0 || ix >= W) continue;
                        float xv = xp[(int64_t)iy * W + ix];
#pragma unroll
                        for (int j = 0; j < FPT; ++j)
                            if (f0 + j < F) acc[j] = fmaf(xv, w[(((int64_t)(f0 + j) * cpg + ic) * k + ky) * k + kx], acc[j]);
                    }
                }
            }
        } else {
            for (int j = 0; j < FPT; ++j) {
                int f = f0 + j;
                if (f >= F) break;
                const int g = f / fpg;
                for (int ic = 0; ic < cpg; ++ic) {
                    const float* xp = x + ((int64_t)b * C + g * cpg + ic) * H * W;
                    for (int ky = 0; ky < k; ++ky) {
                        int iy = oy * sy + ky * dil - pad;
                        if (iy < 0 || iy >= H) continue;
                        for (int kx = 0; kx < k; ++kx) {
                            int ix = ox * sx + kx * dil - pad;
                            if (ix < 0 || ix >= W) continue;
                            acc[j] = fmaf(xp[(int64_t)iy * W + ix], w[(((int64_t)f * cpg + ic) * k + ky) * k + kx], acc[j]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < FPT; ++j)
            if (f0 + j < F) y[(((int64_t)b * F + f0 + j) * OH + oy) * OW + ox] = acc[j];
    }
}

// bias_add / activation / bias_activation: channel = (i / channel_stride) % channels (lightnet-kernels-shared/src/lib.rs:10-40)
__global__ void bias_act_f32_kernel(const float* x, const float* __restrict__ bias, float* y, int64_t n,
                                    int64_t channels, int64_t channel_stride, int act) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float v = x[i];
        if (bias) v += bias[(i / channel_stride) % channels];
        y[i] = ln_act_f32(act, v);
    }
}

__global__ void channel_scale_f32_kernel(const float* __restrict__ x, const float* __restrict__ scale, float* __restrict__ y, int64_t n, int64_t channels,
                                         int64_t channel_stride) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = __fmul_rn(x[i], scale[(i / channel_stride) % channels]);
}

// [region] forward (lightnet-cuda/src/host_ops.rs:73-116): channel-major NCHW entries -> spatial-major [batch, spatial, anchor, entry],
// logistic objectness (entry 4), optional softmax over the class entries.  One thread per (batch, cell, anchor).
__global__ void region_forward_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t batch, int spatial, int anchors, int entries, int classes,
                                          int softmax_classes) {
    const int64_t total = batch * spatial * anchors;
    const int64_t channels = (int64_t)anchors * entries;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int a = (int)(i % anchors);
        const int64_t s = (i / anchors) % spatial, b = i / ((int64_t)anchors * spatial);
        float* out = y + (b * spatial + s) * channels + (int64_t)a * entries;
        const float* in = x + (b * channels + (int64_t)a * entries) * spatial + s;
        for (int e = 0; e < entries; ++e) out[e] = in[(int64_t)e * spatial];
        out[4] = 1.0f / (1.0f + expf(-out[4]));
        if (softmax_classes) {
            float mx = -INFINITY;
            for (int c = 0; c < classes; ++c) mx = fmaxf(mx, out[5 + c]);
            float sum = 0.0f;
            for (int c = 0; c < classes; ++c) {
                const float v = expf(out[5 + c] - mx);
                out[5 + c] = v;
                sum += v;
            }
            if (sum > 0.0f)
                for (int c = 0; c < classes; ++c) out[5 + c] = out[5 + c] / sum;
        }
    }
}

// modern_yolo_forward_f32 (lightnet-cuda/src/lib.rs:4884-4915): every entry sanitised, the trailing 1 + classes planes through a
// sigmoid of the logit clamped to [-30, 30].
__global__ void modern_activate_f32_kernel(const float* __restrict__ x, float* __restrict__ y, long long n, long long spatial, int channels, int class_begin) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)((i / spatial) % channels);
        float v = ln_finite_or_zero(x[i]);
        if (c >= class_begin) v = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-fminf(fmaxf(v, -30.0f), 30.0f))));
        y[i] = v;
    }
}

// modern_yolo_predecode (lightnet-cuda-oxide/src/kernels/dense_loss.rs:788-812): one thread per cell; the softmax expectation of
// each side's bins (modern_yolo/cpu.rs:283-308), corners to a sanitised centre-size box (cpu.rs:340-387), then the objectness
// and class planes copied behind it.
__global__ void modern_predecode_f32_kernel(const float* __restrict__ x, float* __restrict__ y, long long cells, int w, int h, int classes, int coords) {
    const long long s = (long long)w * h;
    const int bins = coords / 4 > 2 ? coords / 4 : 2, cin = coords + 1 + classes, cout = 5 + classes;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < cells; g += (long long)gridDim.x * blockDim.x) {
        const long long b = g / s, loc = g - b * s;
        const float* px = x + b * cin * s + loc;
        float side[4];
        for (int sd = 0; sd < 4; ++sd) {
            float mx = -INFINITY;
            for (int k = 0; k < bins; ++k) mx = fmaxf(mx, ln_finite_or_zero(px[(long long)(sd * bins + k) * s]));
            float denom = 0.0f, expected = 0.0f;
            for (int k = 0; k < bins; ++k) {
                const float e = expf(fminf(fmaxf(__fsub_rn(ln_finite_or_zero(px[(long long)(sd * bins + k) * s]), mx), -60.0f), 60.0f));
                denom = __fadd_rn(denom, e);
                expected = __fadd_rn(expected, __fmul_rn((float)k, e));
            }
            side[sd] = __fdiv_rn(expected, fmaxf(denom, 1e-8f));
        }
        const int row = (int)(loc / w), col = (int)(loc - (long long)row * w);
        const float cx = (float)col + 0.5f, cy = (float)row + 0.5f;
        float left = ln_finite_or_zero(__fdiv_rn(__fsub_rn(cx, side[0]), (float)w)), top = ln_finite_or_zero(__fdiv_rn(__fsub_rn(cy, side[1]), (float)h));
        float right = ln_finite_or_zero(__fdiv_rn(__fadd_rn(cx, side[2]), (float)w)), bottom = ln_finite_or_zero(__fdiv_rn(__fadd_rn(cy, side[3]), (float)h));
        if (right < left) { const float t = left; left = right; right = t; }
        if (bottom < top) { const float t = top; top = bottom; bottom = t; }
        float* py = y + b * cout * s + loc;
        py[0] = ln_finite_or_zero(__fmul_rn(0.5f, __fadd_rn(left, right)));
        py[s] = ln_finite_or_zero(__fmul_rn(0.5f, __fadd_rn(top, bottom)));
        py[2 * s] = fmaxf(ln_finite_or_zero(fmaxf(__fsub_rn(right, left), 1e-6f)), 1e-6f);
        py[3 * s] = fmaxf(ln_finite_or_zero(fmaxf(__fsub_rn(bottom, top), 1e-6f)), 1e-6f);
        for (int e = 0; e < classes + 1; ++e) py[(long long)(4 + e) * s] = px[(long long)(coords + e) * s];
    }
}

// Classic [yolo] head activation on anchor-major NCHW entries (lightnet-cuda/src/lib.rs:4951-4966): logistic on every entry but w / h
// (none when new_coords), then x, y scaled: v * scale_xy - 0.5 * (scale_xy - 1).
__global__ void yolo_activate_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t n, int64_t plane, int entries, float scale_xy,
                                         int new_coords) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int entry = (int)((i / plane) % entries);
        float v = x[i];
        if (!new_coords && entry != 2 && entry != 3) v = 1.0f / (1.0f + expf(-v));
        if (entry < 2) v = __fsub_rn(__fmul_rn(v, scale_xy), __fmul_rn(0.5f, __fsub_rn(scale_xy, 1.0f)));
        y[i] = v;
    }
}

// (tensors start at 512-byte boundaries or at an image of a batch: four values at a time while the count allows)
__global__ void add_f32_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ y, int64_t n) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    const bool vec = ((((uintptr_t)a) | ((uintptr_t)b) | ((uintptr_t)y)) & 15) == 0;
    const int64_t n4 = vec ? n / 4 : 0;
    for (int64_t i = t; i < n4; i += step) {
        const float4 u = reinterpret_cast<const float4*>(a)[i], v = reinterpret_cast<const float4*>(b)[i];
        reinterpret_cast<float4*>(y)[i] = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
    }
    for (int64_t i = 4 * n4 + t; i < n; i += step) y[i] = a[i] + b[i];
}

// shortcut_fit: flat per-sample crop / zero-pad (lightnet-cuda/src/lib.rs:4036-4056)
__global__ void shortcut_fit_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t batch, int64_t in_len,
                                        int64_t out_len) {
    int64_t n = batch * out_len;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t b = i / out_len, j = i % out_len;
        y[i] = j < in_len ? x[b * in_len + j] : 0.0f;
    }
}

// route copy of one source's channel slice (runtime/layer_ops.rs:1850-1883): per image one contiguous run of `run` floats.
// blockIdx.y = image.  (With a 64-bit division per value the copies of YOLOv4 608 x 608 took 333 us per image.)
__global__ void route_copy_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t run, int64_t x_image, int64_t y_image) {
    const float* src = x + blockIdx.y * x_image;
    float* dst = y + blockIdx.y * y_image;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    const int64_t n4 = ((((uintptr_t)src) | ((uintptr_t)dst)) & 15) == 0 ? run / 4 : 0;
    for (int64_t i = t; i < n4; i += step) reinterpret_cast<float4*>(dst)[i] = __ldg(reinterpret_cast<const float4*>(src) + i);
    for (int64_t i = 4 * n4 + t; i < run; i += step) dst[i] = src[i];
}

// Darknet max-pool: window origin o*stride - padding/2, taps outside skipped, start at -inf
// (runtime/layer_ops.rs:1740-1799; lightnet-kernels-shared/src/lib.rs:95-140)
__global__ void maxpool_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t BC, int H, int W, int OH, int OW,
                                   int size, int sx, int sy, int padding) {
    int64_t n = BC * OH * OW;
    const int off = padding / 2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int ox = (int)(i % OW), oy = (int)((i / OW) % OH);
        int64_t bc = i / ((int64_t)OW * OH);
        const float* xp = x + bc * H * W;
        float m = -INFINITY;
        for (int ky = 0; ky < size; ++ky) {
            int iy = oy * sy + ky - off;
            if (iy < 0 || iy >= H) continue;
            for (int kx = 0; kx < size; ++kx) {
                int ix = ox * sx + kx - off;
                if (ix < 0 || ix >= W) continue;
                m = fmaxf(m, xp[(int64_t)iy * W + ix]);
            }
        }
        y[i] = m;
    }
}

// nearest up-sample: out[y,x] = scale * in[y/s, x/s] (runtime/layer_ops.rs:2208-2256)
__global__ void upsample_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t BC, int H, int W, int s, float scale) {
    const int OH = H * s, OW = W * s;
    int64_t n = BC * OH * OW;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int ox = (int)(i % OW), oy = (int)((i / OW) % OH);
        int64_t bc = i / ((int64_t)OW * OH);
        y[i] = scale * x[(bc * H + oy / s) * W + ox / s];
    }
}

// reverse up-sample: out[y/s, x/s] += scale * in[y, x]; gather form (each output sums its s*s block in the
// row-major order the reference visits them)
__global__ void upsample_reverse_f32_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t BC, int H, int W, int s,
                                            float scale) {
    const int OH = H / s, OW = W / s;
    int64_t n = BC * OH * OW;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int ox = (int)(i % OW), oy = (int)((i / OW) % OH);
        int64_t bc = i / ((int64_t)OW * OH);
        float acc = 0.0f;
        for (int dy = 0; dy < s; ++dy)
            for (int dx = 0; dx < s; ++dx) acc += scale * x[(bc * H + oy * s + dy) * W + ox * s + dx];
        y[i] = acc;
    }
}

__global__ void bn_fold_kernel(const float* gamma, const float* mean, const float* var, const float* bias, float eps, float* scale,
                               float* bias_out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // single IEEE operations in the order of weights_io.rs:32-92 (no fused multiply-add), so the result has the host fold's bits
    float s = __fdiv_rn(gamma[i], __fsqrt_rn(__fadd_rn(var[i], eps)));
    scale[i] = s;
    bias_out[i] = __fsub_rn(bias[i], __fmul_rn(mean[i], s));
}

int grid_for(ln_ctx* ctx, int64_t n) {
    int64_t b = (n + kThreads - 1) / kThreads;
    int64_t cap = (int64_t)ctx->sm_count * 32;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

bool is_f32(const ln_tensor* t) { return t && t->dtype == LN_F32; }

template <class K>
cudaError_t launch_conv_f32(ln_ctx* ctx, K kernel, const ConvF32& p, int threads, size_t smem, dim3 grid) {
    if (smem > 48 * 1024 && !ctx->configured_kernels.count((const void*)kernel)) {  // once per kernel per context
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        ctx->configured_kernels.insert((const void*)kernel);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ctx->launches++;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

// 1: 1x1 without padding, 3: 3x3 without dilation, 0: any other kernel.
int conv_f32_kind(int k, int pad, int dil) { return k == 1 && pad == 0 ? 1 : (k == 3 && dil == 1 ? 3 : 0); }

// Ungrouped convolution with optional bias and activation, cut as ln_conv_f32_choose says.
int conv_f32_run(ln_ctx* ctx, ConvF32 p, bool one_chain, const char* who) {
    const int64_t NP = (int64_t)p.B * p.OH * p.OW;
    const int ks = conv_f32_kind(p.k, p.pad, p.dil);
    const bool async = ks != 0 && p.F > 32 && (p.K & 3) == 0 && (((uintptr_t)p.w) & 15) == 0;
    const ln_conv_f32_cut cut = ln_conv_f32_choose(ctx->sm_count, p.B, (int64_t)p.OH * p.OW, p.F, p.K, ks, async, one_chain);
    const bool wide = async && cut.bn == 128, narrow = cut.bm == 32;
    const dim3 grid((unsigned)((NP + cut.bn - 1) / cut.bn), (unsigned)((p.F + cut.bm - 1) / cut.bm), (unsigned)cut.parts);
    cudaError_t e;
    if (wide) e = ks == 1 ? launch_conv_f32(ctx, conv2d_f32_async_kernel<128, 1>, p, 128, sizeof(ConvF32Shared<128, 1>), grid)
                          : launch_conv_f32(ctx, conv2d_f32_async_kernel<128, 3>, p, 128, sizeof(ConvF32Shared<128, 3>), grid);
    else if (async) e = ks == 1 ? launch_conv_f32(ctx, conv2d_f32_async_kernel<64, 1>, p, 64, sizeof(ConvF32Shared<64, 1>), grid)
                                : launch_conv_f32(ctx, conv2d_f32_async_kernel<64, 3>, p, 64, sizeof(ConvF32Shared<64, 3>), grid);
    else if (narrow) e = ks == 1 ? launch_conv_f32(ctx, conv2d_f32_gemm_kernel<32, 128, 1>, p, 64, 0, grid)
                                 : (ks == 3 ? launch_conv_f32(ctx, conv2d_f32_gemm_kernel<32, 128, 3>, p, 64, 0, grid) : launch_conv_f32(ctx, conv2d_f32_gemm_kernel<32, 128, 0>, p, 64, 0, grid));
    else e = ks == 1 ? launch_conv_f32(ctx, conv2d_f32_gemm_kernel<64, 64, 1>, p, 64, 0, grid)
                     : (ks == 3 ? launch_conv_f32(ctx, conv2d_f32_gemm_kernel<64, 64, 3>, p, 64, 0, grid) : launch_conv_f32(ctx, conv2d_f32_gemm_kernel<64, 64, 0>, p, 64, 0, grid));
    if (e == cudaSuccess) return LN_OK;
    (void)cudaGetLastError();  // (the next launch is checked for its own error)
    return ln_fail(ctx, LN_ERR_CUDA, "%s launch: %s", who, cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int32_t ln_conv2d_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* weights, const int64_t output_shape[4],
                      int64_t input_channels, int64_t input_height, int64_t input_width, int64_t filters, int64_t kernel_size,
                      int64_t stride_x, int64_t stride_y, int64_t dilation, int64_t padding, int64_t groups, ln_tensor** out) {
    return ln_conv2d_bias_act_f32(ctx, x, weights, nullptr, output_shape, input_channels, input_height, input_width, filters, kernel_size, stride_x, stride_y, dilation,
                                  padding, groups, LN_ACT_LINEAR, false, out);
}

}  // extern "C"

// conv2d_f32 followed by bias_activation_f32 (bias may be null) without the pass over memory between them
int ln_conv2d_bias_act_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* weights, const ln_tensor* bias, const int64_t output_shape[4], int64_t input_channels,
                           int64_t input_height, int64_t input_width, int64_t filters, int64_t kernel_size, int64_t stride_x, int64_t stride_y, int64_t dilation,
                           int64_t padding, int64_t groups, int activation, bool one_chain, ln_tensor** out) {
    if (!ctx || !out || !output_shape) return ln_fail(ctx, LN_ERR_ARG, "ln_conv2d_f32: NULL argument");
    if (!is_f32(x) || !is_f32(weights)) return ln_fail(ctx, LN_ERR_ARG, "ln_conv2d_f32: f32 tensors required");
    if (groups < 1 || filters % groups || input_channels % groups || kernel_size < 1 || stride_x < 1 || stride_y < 1 || dilation < 1)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_conv2d_f32: invalid geometry (groups %lld filters %lld channels %lld)", (long long)groups,
                       (long long)filters, (long long)input_channels);
    if (x->c != input_channels || x->h != input_height || x->w != input_width)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_conv2d_f32: input tensor is [%lld,%lld,%lld,%lld], geometry says C=%lld H=%lld W=%lld",
                       (long long)x->n, (long long)x->c, (long long)x->h, (long long)x->w, (long long)input_channels,
                       (long long)input_height, (long long)input_width);
    if (weights->count() != filters * (input_channels / groups) * kernel_size * kernel_size)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_conv2d_f32: weight tensor has %lld elements, expected %lld", (long long)weights->count(),
                       (long long)(filters * (input_channels / groups) * kernel_size * kernel_size));
    // lightnet-model model.rs:6472 conv_dim (dilation does not enter the extent)
    int64_t oh = (input_height + 2 * padding - kernel_size < 0 ? 0 : input_height + 2 * padding - kernel_size) / stride_y + 1;
    int64_t ow = (input_width + 2 * padding - kernel_size < 0 ? 0 : input_width + 2 * padding - kernel_size) / stride_x + 1;
    if (output_shape[0] != x->n || output_shape[1] != filters || output_shape[2] != oh || output_shape[3] != ow)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_conv2d_f32: output_shape [%lld,%lld,%lld,%lld] does not match [%lld,%lld,%lld,%lld]",
                       (long long)output_shape[0], (long long)output_shape[1], (long long)output_shape[2], (long long)output_shape[3],
                       (long long)x->n, (long long)filters, (long long)oh, (long long)ow);
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, filters, oh, ow);
    if (!y) return LN_ERR_CUDA;
    const float* b = bias ? (const float*)bias->ptr : nullptr;
    int rc = LN_OK;
    const int ks = conv_f32_kind((int)kernel_size, (int)padding, (int)dilation);
    if (groups == 1 && ln_conv_f32_blocked(x->n, input_channels, input_height, input_width, filters, kernel_size, oh, ow) &&
        !ln_conv_f32_per_tap(x->n, oh * ow, filters, input_channels * kernel_size * kernel_size, ks, b || activation != LN_ACT_LINEAR)) {
        ConvF32 p = {};
        p.x = (const float*)x->ptr; p.w = (const float*)weights->ptr; p.bias = b; p.y = (float*)y->ptr;
        p.B = (int)x->n; p.C = (int)input_channels; p.H = (int)input_height; p.W = (int)input_width; p.F = (int)filters; p.k = (int)kernel_size;
        p.sx = (int)stride_x; p.sy = (int)stride_y; p.dil = (int)dilation; p.pad = (int)padding; p.OH = (int)oh; p.OW = (int)ow;
        p.K = (int)(input_channels * kernel_size * kernel_size);
        p.act = activation;
        rc = conv_f32_run(ctx, p, one_chain, "conv2d_f32");
    } else {
        int64_t total = x->n * ((filters + 3) / 4) * oh * ow;
        conv2d_f32_kernel<4><<<grid_for(ctx, total), kThreads, 0, ctx->stream>>>(
            (const float*)x->ptr, (const float*)weights->ptr, (float*)y->ptr, (int)x->n, (int)input_channels, (int)input_height,
            (int)input_width, (int)filters, (int)kernel_size, (int)stride_x, (int)stride_y, (int)dilation, (int)padding, (int)groups,
            (int)oh, (int)ow);
        ctx->launches++;
        if (b || activation != LN_ACT_LINEAR) {
            bias_act_f32_kernel<<<grid_for(ctx, y->count()), kThreads, 0, ctx->stream>>>((const float*)y->ptr, b, (float*)y->ptr, y->count(), filters, oh * ow, activation);
            ctx->launches++;
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = ln_fail(ctx, LN_ERR_CUDA, "conv2d_f32 launch: %s", cudaGetErrorString(e));
    }
    if (rc) { ln_tensor_release(y); return rc; }
    *out = y;
    return LN_OK;
}

extern "C" {

static int32_t bias_act_impl(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* bias, int64_t channels, int64_t channel_stride,
                             int32_t activation, ln_tensor** out, const char* who) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "%s: NULL argument", who);
    if (!is_f32(x) || (bias && !is_f32(bias))) return ln_fail(ctx, LN_ERR_ARG, "%s: f32 tensors required", who);
    if (bias && (channels < 1 || channel_stride < 1 || bias->count() != channels))
        return ln_fail(ctx, LN_ERR_SHAPE, "%s: bias has %lld elements for %lld channels", who, (long long)bias->count(), (long long)channels);
    if (activation < LN_ACT_LINEAR || activation > LN_ACT_RELU) return ln_fail(ctx, LN_ERR_UNSUPPORTED, "%s: activation %d is not on the detector path", who, activation);
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);
    if (!y) return LN_ERR_CUDA;
    bias_act_f32_kernel<<<grid_for(ctx, x->count()), kThreads, 0, ctx->stream>>>(
        (const float*)x->ptr, bias ? (const float*)bias->ptr : nullptr, (float*)y->ptr, x->count(), channels > 0 ? channels : 1,
        channel_stride > 0 ? channel_stride : 1, activation);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "%s launch: %s", who, cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_bias_add_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* bias, int64_t channels, int64_t channel_stride, ln_tensor** out) {
    if (!bias) return ln_fail(ctx, LN_ERR_ARG, "ln_bias_add_f32: bias is NULL");
    return bias_act_impl(ctx, x, bias, channels, channel_stride, LN_ACT_LINEAR, out, "ln_bias_add_f32");
}
int32_t ln_activation_f32(ln_ctx* ctx, const ln_tensor* x, int32_t activation, ln_tensor** out) {
    return bias_act_impl(ctx, x, nullptr, 1, 1, activation, out, "ln_activation_f32");
}
int32_t ln_bias_activation_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* bias, int64_t channels, int64_t channel_stride,
                               int32_t activation, ln_tensor** out) {
    if (!bias) return ln_fail(ctx, LN_ERR_ARG, "ln_bias_activation_f32: bias is NULL");
    return bias_act_impl(ctx, x, bias, channels, channel_stride, activation, out, "ln_bias_activation_f32");
}

int32_t ln_channel_scale_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* scale, int64_t channels, int64_t channel_stride, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_channel_scale_f32: NULL argument");
    if (!is_f32(x) || !is_f32(scale)) return ln_fail(ctx, LN_ERR_ARG, "ln_channel_scale_f32: f32 tensors required");
    if (channels < 1 || channel_stride < 1 || scale->count() != channels)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_channel_scale_f32: scale has %lld elements for %lld channels", (long long)scale->count(), (long long)channels);
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);
    if (!y) return LN_ERR_CUDA;
    channel_scale_f32_kernel<<<grid_for(ctx, x->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (const float*)scale->ptr, (float*)y->ptr, x->count(), channels, channel_stride);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "channel_scale launch: %s", cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_region_forward_f32(ln_ctx* ctx, const ln_tensor* x, int64_t anchors, int64_t entries, int64_t classes, int32_t softmax_classes, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_region_forward_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_region_forward_f32: f32 tensor required");
    if (anchors < 1 || classes < 0 || entries < classes + 5 || x->c != anchors * entries)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_region_forward_f32: %lld channels do not hold %lld anchors of %lld entries (>= classes + 5)", (long long)x->c, (long long)anchors, (long long)entries);
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);  // same element count; the layout is [batch, spatial, anchor, entry]
    if (!y) return LN_ERR_CUDA;
    region_forward_f32_kernel<<<grid_for(ctx, x->n * x->h * x->w * anchors), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)y->ptr, x->n, (int)(x->h * x->w), (int)anchors,
                                                                                                         (int)entries, (int)classes, softmax_classes);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "region_forward launch: %s", cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_yolo_activate_f32(ln_ctx* ctx, const ln_tensor* x, int64_t classes, float scale_xy, int32_t new_coords, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_yolo_activate_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_yolo_activate_f32: f32 tensor required");
    if (classes < 0 || x->c % (classes + 5)) return ln_fail(ctx, LN_ERR_SHAPE, "YOLO head tensor length mismatch: %lld channels are not a multiple of %lld entries", (long long)x->c, (long long)(classes + 5));
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);
    if (!y) return LN_ERR_CUDA;
    yolo_activate_f32_kernel<<<grid_for(ctx, x->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)y->ptr, x->count(), x->h * x->w, (int)(classes + 5), scale_xy, new_coords);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "yolo_activate launch: %s", cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_modern_yolo_forward_f32(ln_ctx* ctx, const ln_tensor* x, int64_t classes, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_forward_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_forward_f32: f32 tensor required");
    if (classes < 0) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_forward_f32: negative class count");
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);
    if (!y) return LN_ERR_CUDA;
    const long long class_begin = x->c - (classes + 1) > 0 ? x->c - (classes + 1) : 0;  // saturating_sub, lib.rs:4898
    modern_activate_f32_kernel<<<grid_for(ctx, x->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)y->ptr, x->count(), x->h * x->w, (int)x->c, (int)class_begin);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "modern_yolo_forward launch: %s", cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_modern_yolo_predecode_f32(ln_ctx* ctx, const ln_tensor* x, int64_t classes, int64_t coords, int32_t kind, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_predecode_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_predecode_f32: f32 tensor required");
    if (kind != 1 && kind != 2) return ln_fail(ctx, LN_ERR_UNSUPPORTED, "ln_modern_yolo_predecode_f32: kind %d is not a distribution head (1 = ppyoloe, 2 = yolonas)", kind);
    if (classes < 1 || coords < 8 || coords % 4) return ln_fail(ctx, LN_ERR_ARG, "ln_modern_yolo_predecode_f32: %lld classes, %lld box entries", (long long)classes, (long long)coords);
    if (x->c != coords + 1 + classes) return ln_fail(ctx, LN_ERR_SHAPE, "distribution head tensor length mismatch: %lld channels, expected %lld", (long long)x->c, (long long)(coords + 1 + classes));
    cudaSetDevice(ctx->device);
    ln_tensor* y = ln_tensor_new(ctx, LN_F32, x->n, 5 + classes, x->h, x->w);
    if (!y) return LN_ERR_CUDA;
    const long long cells = x->n * x->h * x->w;
    modern_predecode_f32_kernel<<<grid_for(ctx, cells), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)y->ptr, cells, (int)x->w, (int)x->h, (int)classes, (int)coords);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(y); return ln_fail(ctx, LN_ERR_CUDA, "modern_yolo_predecode launch: %s", cudaGetErrorString(e)); }
    *out = y;
    return LN_OK;
}

int32_t ln_shortcut_add_f32(ln_ctx* ctx, const ln_tensor* x, const ln_tensor* y, ln_tensor** out) {
    if (!ctx || !out) return ln_fail(ctx, LN_ERR_ARG, "ln_shortcut_add_f32: NULL argument");
    if (!is_f32(x) || !is_f32(y)) return ln_fail(ctx, LN_ERR_ARG, "ln_shortcut_add_f32: f32 tensors required");
    if (x->count() != y->count()) return ln_fail(ctx, LN_ERR_SHAPE, "ln_shortcut_add_f32: %lld vs %lld elements", (long long)x->count(), (long long)y->count());
    cudaSetDevice(ctx->device);
    ln_tensor* o = ln_tensor_new(ctx, LN_F32, x->n, x->c, x->h, x->w);
    if (!o) return LN_ERR_CUDA;
    add_f32_kernel<<<grid_for(ctx, x->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (const float*)y->ptr, (float*)o->ptr, x->count());
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(o); return ln_fail(ctx, LN_ERR_CUDA, "shortcut_add launch: %s", cudaGetErrorString(e)); }
    *out = o;
    return LN_OK;
}

int32_t ln_shortcut_fit_f32(ln_ctx* ctx, const ln_tensor* x, int64_t batch, const int64_t output_shape[4], ln_tensor** out) {
    if (!ctx || !out || !output_shape) return ln_fail(ctx, LN_ERR_ARG, "ln_shortcut_fit_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_shortcut_fit_f32: f32 tensor required");
    if (batch < 1 || x->count() % batch || output_shape[0] != batch) return ln_fail(ctx, LN_ERR_SHAPE, "ln_shortcut_fit_f32: batch %lld does not divide the tensors", (long long)batch);
    cudaSetDevice(ctx->device);
    ln_tensor* o = ln_tensor_new(ctx, LN_F32, output_shape[0], output_shape[1], output_shape[2], output_shape[3]);
    if (!o) return LN_ERR_CUDA;
    shortcut_fit_f32_kernel<<<grid_for(ctx, o->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)o->ptr, batch,
                                                                                    x->count() / batch, o->count() / batch);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(o); return ln_fail(ctx, LN_ERR_CUDA, "shortcut_fit launch: %s", cudaGetErrorString(e)); }
    *out = o;
    return LN_OK;
}

int32_t ln_route_concat_f32(ln_ctx* ctx, const ln_tensor* const* inputs, int32_t n_inputs, const int64_t* input_channel_offsets,
                            const int64_t* input_channels, const int64_t* input_total_channels, const int64_t output_shape[4],
                            int64_t channel_stride, ln_tensor** out) {
    if (!ctx || !out || !inputs || !input_channel_offsets || !input_channels || !input_total_channels || !output_shape || n_inputs < 1)
        return ln_fail(ctx, LN_ERR_ARG, "ln_route_concat_f32: NULL argument");
    int64_t sum = 0;
    for (int i = 0; i < n_inputs; ++i) {
        if (!is_f32(inputs[i])) return ln_fail(ctx, LN_ERR_ARG, "ln_route_concat_f32: input %d is not f32", i);
        if (inputs[i]->c != input_total_channels[i] || input_channel_offsets[i] + input_channels[i] > input_total_channels[i] ||
            inputs[i]->h * inputs[i]->w != channel_stride || inputs[i]->n != output_shape[0])
            return ln_fail(ctx, LN_ERR_SHAPE, "ln_route_concat_f32: input %d does not match its channel slice / plane size", i);
        sum += input_channels[i];
    }
    if (sum != output_shape[1] || output_shape[2] * output_shape[3] != channel_stride)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_route_concat_f32: slices sum to %lld channels, output has %lld", (long long)sum, (long long)output_shape[1]);
    cudaSetDevice(ctx->device);
    ln_tensor* o = ln_tensor_new(ctx, LN_F32, output_shape[0], output_shape[1], output_shape[2], output_shape[3]);
    if (!o) return LN_ERR_CUDA;
    int64_t c0 = 0;
    for (int i = 0; i < n_inputs; ++i) {
        const int64_t run = input_channels[i] * channel_stride;
        for (int64_t b0 = 0; b0 < o->n; b0 += 65535) {  // (grid limit in y)
            const int64_t images = o->n - b0 < 65535 ? o->n - b0 : 65535, x_image = input_total_channels[i] * channel_stride, y_image = o->c * channel_stride;
            route_copy_f32_kernel<<<dim3((unsigned)grid_for(ctx, (run + 3) / 4), (unsigned)images), kThreads, 0, ctx->stream>>>(
                (const float*)inputs[i]->ptr + b0 * x_image + input_channel_offsets[i] * channel_stride, (float*)o->ptr + b0 * y_image + c0 * channel_stride, run, x_image, y_image);
        }
        ctx->launches++;
        c0 += input_channels[i];
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(o); return ln_fail(ctx, LN_ERR_CUDA, "route_concat launch: %s", cudaGetErrorString(e)); }
    *out = o;
    return LN_OK;
}

int32_t ln_maxpool_f32(ln_ctx* ctx, const ln_tensor* x, const int64_t output_shape[4], int64_t channels, int64_t input_height,
                       int64_t input_width, int64_t size, int64_t stride_x, int64_t stride_y, int64_t padding, ln_tensor** out) {
    if (!ctx || !out || !output_shape) return ln_fail(ctx, LN_ERR_ARG, "ln_maxpool_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_maxpool_f32: f32 tensor required");
    if (x->c != channels || x->h != input_height || x->w != input_width || size < 1 || stride_x < 1 || stride_y < 1)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_maxpool_f32: geometry does not match the input tensor");
    // lightnet-model model.rs:8854 pool_dim
    int64_t oh = (input_height + padding - size < 0 ? 0 : input_height + padding - size) / stride_y + 1;
    int64_t ow = (input_width + padding - size < 0 ? 0 : input_width + padding - size) / stride_x + 1;
    if (output_shape[0] != x->n || output_shape[1] != channels || output_shape[2] != oh || output_shape[3] != ow)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_maxpool_f32: output_shape does not match pool_dim (%lld x %lld)", (long long)oh, (long long)ow);
    cudaSetDevice(ctx->device);
    ln_tensor* o = ln_tensor_new(ctx, LN_F32, x->n, channels, oh, ow);
    if (!o) return LN_ERR_CUDA;
    maxpool_f32_kernel<<<grid_for(ctx, o->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)o->ptr, x->n * channels,
                                                                                (int)input_height, (int)input_width, (int)oh, (int)ow,
                                                                                (int)size, (int)stride_x, (int)stride_y, (int)padding);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(o); return ln_fail(ctx, LN_ERR_CUDA, "maxpool launch: %s", cudaGetErrorString(e)); }
    *out = o;
    return LN_OK;
}

int32_t ln_upsample_f32(ln_ctx* ctx, const ln_tensor* x, const int64_t output_shape[4], int64_t channels, int64_t input_height,
                        int64_t input_width, int64_t stride, float scale, int32_t reverse, ln_tensor** out) {
    if (!ctx || !out || !output_shape) return ln_fail(ctx, LN_ERR_ARG, "ln_upsample_f32: NULL argument");
    if (!is_f32(x)) return ln_fail(ctx, LN_ERR_ARG, "ln_upsample_f32: f32 tensor required");
    if (stride < 1) return ln_fail(ctx, LN_ERR_SHAPE, "ln_upsample_f32: upsample stride cannot be zero");
    if (x->c != channels || x->h != input_height || x->w != input_width)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_upsample_f32: geometry does not match the input tensor");
    int64_t oh = reverse ? input_height / stride : input_height * stride;
    int64_t ow = reverse ? input_width / stride : input_width * stride;
    if (output_shape[0] != x->n || output_shape[1] != channels || output_shape[2] != oh || output_shape[3] != ow)
        return ln_fail(ctx, LN_ERR_SHAPE, "ln_upsample_f32: output_shape does not match (%lld x %lld)", (long long)oh, (long long)ow);
    cudaSetDevice(ctx->device);
    ln_tensor* o = ln_tensor_new(ctx, LN_F32, x->n, channels, oh, ow);
    if (!o) return LN_ERR_CUDA;
    if (reverse)
        upsample_reverse_f32_kernel<<<grid_for(ctx, o->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)o->ptr,
                                                                                             x->n * channels, (int)input_height,
                                                                                             (int)input_width, (int)stride, scale);
    else
        upsample_f32_kernel<<<grid_for(ctx, o->count()), kThreads, 0, ctx->stream>>>((const float*)x->ptr, (float*)o->ptr, x->n * channels,
                                                                                     (int)input_height, (int)input_width, (int)stride, scale);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(o); return ln_fail(ctx, LN_ERR_CUDA, "upsample launch: %s", cudaGetErrorString(e)); }
    *out = o;
    return LN_OK;
}

int32_t ln_batchnorm_fold_f32(ln_ctx* ctx, const ln_tensor* gamma, const ln_tensor* mean, const ln_tensor* variance,
                              const ln_tensor* bias, float eps, ln_tensor** scale_out, ln_tensor** bias_out) {
    if (!ctx || !scale_out || !bias_out) return ln_fail(ctx, LN_ERR_ARG, "ln_batchnorm_fold_f32: NULL argument");
    if (!is_f32(gamma) || !is_f32(mean) || !is_f32(variance) || !is_f32(bias)) return ln_fail(ctx, LN_ERR_ARG, "ln_batchnorm_fold_f32: f32 tensors required");
    int64_t n = gamma->count();
    if (mean->count() != n || variance->count() != n || bias->count() != n) return ln_fail(ctx, LN_ERR_SHAPE, "ln_batchnorm_fold_f32: parameter length mismatch for %lld filters", (long long)n);
    cudaSetDevice(ctx->device);
    ln_tensor* s = ln_tensor_new(ctx, LN_F32, 1, n, 1, 1);
    ln_tensor* b = ln_tensor_new(ctx, LN_F32, 1, n, 1, 1);
    if (!s || !b) { ln_tensor_release(s); ln_tensor_release(b); return LN_ERR_CUDA; }
    bn_fold_kernel<<<blocks_for(n), kThreads, 0, ctx->stream>>>((const float*)gamma->ptr, (const float*)mean->ptr, (const float*)variance->ptr,
                                                                (const float*)bias->ptr, eps, (float*)s->ptr, (float*)b->ptr, (int)n);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { ln_tensor_release(s); ln_tensor_release(b); return ln_fail(ctx, LN_ERR_CUDA, "bn_fold launch: %s", cudaGetErrorString(e)); }
    *scale_out = s;
    *bias_out = b;
    return LN_OK;
}

}  // extern "C"
