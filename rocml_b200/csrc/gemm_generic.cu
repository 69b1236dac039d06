// Plain tiled matrix product on the CUDA cores: out[M, N] = x[M, K] . W[N, K]^T (+ bias[N], 32-bit).
//
// 32-bit FMA accumulation, no tensor cores and no reduced-precision mode, for every element
// type.  It is the matrix product of the true 32-bit path, the fallback for sizes the
// tcgen05 kernel refuses, and the reference the tcgen05 kernel is tested against.  It stands
// where the reference has gemv_f16 / gemm_xwt_f16 (rocml-kernels/kernels/gemv_f16.hip:8-36,
// gemm_f16.hip:10-41).  Three kernels, and in each the order in which a row's products are added
// depends on the weight's sizes alone: a row's result does not depend on what else is in the batch (up to 16 rows, or 17
// to any number), so that a prompt in pieces gives the same bits as the whole.
//
// * The tiled kernels take any type, layout and size: k ascending.
//
// * Few rows of 32-bit operands (up to 16, a decode step of the 32-bit path) are bound
//   by reading the weight once: a warp owns two weight rows and streams them with 16-byte loads, every
//   lane multiplying its slice of k with the same slice of all the step's rows (which a block brings
//   into shared memory tile by tile), and the lanes' sums meet in a shuffle tree.
//
// * More rows of 32-bit operands whose rows start on 16 bytes: tiles in a pipeline, the sum over k in up to eight
//   stretches that are added as a tree, whether the blocks of a cluster have one each or one block has them all.
#include "common.cuh"
#include "sm100.cuh"
#include "api.h"
#include "per_device.h"
#include <algorithm>

using namespace rb;

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename XT, typename WT, typename OT>
__global__ void __launch_bounds__(256)
gemm_tn_kernel(const XT* __restrict__ x, const WT* __restrict__ w, const float* __restrict__ bias,
               OT* __restrict__ out, int M, int N, int K, long long ldx, long long ldo) {
    pdl_trigger();
    pdl_wait();
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int ty = tid / 16, tx = tid % 16;
    const int lr = tid / 4, lc = (tid % 4) * 4;  // this thread loads row lr, k columns lc..lc+3
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lc + j;
            const int m = m0 + lr, n = n0 + lr;
            xs[lc + j][lr] = (m < M && k < K) ? to_f32(x[(size_t)m * ldx + k]) : 0.f;
            ws[lc + j][lr] = (n < N && k < K) ? to_f32(w[(size_t)n * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            out[(size_t)m * ldo + n] = from_f32<OT>(v);
        }
    }
}

// ---- many rows: 128 x 128 tiles, 8 x 8 outputs a thread ------------------------------------------------
// The same sum in the same order (k ascending for every output element) on larger tiles: a thread owns
// two groups of four rows and two groups of four columns (64 apart, so that a warp's 16-byte reads of
// shared memory fall on consecutive banks), a tile of k is 16 deep, and the next tile's global loads are
// in flight while this one is multiplied.  2.5 times the small tiles' rate on a prompt of 2,048 tokens.
constexpr int LBM = 128, LBN = 128, LBK = 16, LLD = LBM + 4;

template <typename XT, typename WT, typename OT>
__global__ void __launch_bounds__(256, 2)
gemm_tn_large_kernel(const XT* __restrict__ x, const WT* __restrict__ w, const float* __restrict__ bias,
                     OT* __restrict__ out, int M, int N, int K, long long ldx, long long ldo) {
    pdl_trigger();
    pdl_wait();
    __shared__ __align__(16) float xs[2][LBK][LLD];
    __shared__ __align__(16) float ws[2][LBK][LLD];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * LBM, n0 = blockIdx.x * LBN;
    const int ty = tid / 16, tx = tid % 16;
    // loads: thread t brings k columns lc .. lc + 3 of rows lr and lr + 64 of both operands
    const int lr = tid / 4, lc = (tid % 4) * 4;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    float xr[2][4], wr[2][4];
    // 32-bit operands whose rows start on 16 bytes are read four k at a time
    const bool x4 = sizeof(XT) == 4 && (ldx & 3) == 0 && ((uintptr_t)x & 15) == 0;
    const bool w4 = sizeof(WT) == 4 && (K & 3) == 0 && ((uintptr_t)w & 15) == 0;
    auto fetch = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = m0 + lr + h * 64, n = n0 + lr + h * 64;
            const int k = k0 + lc;
            if (x4 && m < M && k + 3 < K) {
                const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + (size_t)m * ldx + k);
                xr[h][0] = v.x; xr[h][1] = v.y; xr[h][2] = v.z; xr[h][3] = v.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) xr[h][j] = (m < M && k + j < K) ? to_f32(x[(size_t)m * ldx + k + j]) : 0.f;
            }
            if (w4 && n < N && k + 3 < K) {
                const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + (size_t)n * K + k);
                wr[h][0] = v.x; wr[h][1] = v.y; wr[h][2] = v.z; wr[h][3] = v.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) wr[h][j] = (n < N && k + j < K) ? to_f32(w[(size_t)n * K + k + j]) : 0.f;
            }
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                xs[buf][lc + j][lr + h * 64] = xr[h][j];
                ws[buf][lc + j][lr + h * 64] = wr[h][j];
            }
    };
    fetch(0);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += LBK, buf ^= 1) {
        if (k0 + LBK < K) fetch(k0 + LBK);
#pragma unroll
        for (int kk = 0; kk < LBK; ++kk) {
            float a[8], b[8];
            const float4 a0 = *reinterpret_cast<const float4*>(&xs[buf][kk][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&xs[buf][kk][64 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4*>(&ws[buf][kk][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4*>(&ws[buf][kk][64 + tx * 4]);
            a[0] = a0.x; a[1] = a0.y; a[2] = a0.z; a[3] = a0.w; a[4] = a1.x; a[5] = a1.y; a[6] = a1.z; a[7] = a1.w;
            b[0] = b0.x; b[1] = b0.y; b[2] = b0.z; b[3] = b0.w; b[4] = b1.x; b[5] = b1.y; b[6] = b1.z; b[7] = b1.w;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (k0 + LBK < K) stash(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + j - 4);
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            out[(size_t)m * ldo + n] = from_f32<OT>(v);
        }
    }
}

// ---- more than 16 rows of 32-bit operands: tiles in a pipeline, k split over a cluster --------------------
// Bound by the FMA lanes (128 a multiprocessor) once they have work: a prompt of a few hundred tokens has fewer
// large tiles than the device has multiprocessors, and the plain tiles above ran such products at 10 TFLOP/s.
// So the tiles are lower (32 or 64 rows: 181 rows are 3 x 64, not 2 x 128), and the sum over k is split over the
// blocks of a thread-block cluster until about two blocks a multiprocessor are at work; the parts meet in shared
// memory, so that no partial sums go through global memory and the result is one piece.
// How many parts are best depends on the step's rows, but a row's result must not: k is always cut into the same
// stretches (`f32_stretches`, by the weight's sizes alone), each is summed from zero, and the sums are added as a balanced tree.  A block
// has one, two, four or all of them, an aligned subtree; it keeps finished subtrees that wait for their other half in local memory
// (64 values a thread and level, touched once a stretch).
// Tiles of 32 k arrive by cp.async in their own layout (rows of 36 floats: eight neighbouring rows' 16-byte groups
// fall on different banks), three stages deep.  A thread owns 8 x 8 (BM = 64) or 8 x 4 outputs, rows and columns
// interleaved over the warp so that a warp's 16-byte read is 4 or 8 different groups; a 16-byte group is two
// pairs of k, and each accumulator is a pair (even k, odd k) fed by the two-FMA instruction, so nothing is
// packed or transposed anywhere.  At K = 2,048, the plain tiles and these: 64 x 4,096 135 and 34 us, 181 x 8,192 338 and 167,
// 500 x 2,048 221 and 117, 2,048 x 2,048 398 and 384, 4,096 x 4,096 1,562 and 1,478 (46 TFLOP/s); their error against 64 bits 8e-7 and 2e-7
// (6e-7 where k is one stretch).  With the order of the additions left to the number of parts the last was 1,397.
constexpr int FBN = 128, FBK = 32, FLD = FBK + 4, FSTAGES = 3, FTHREADS = 128;
template <int BM_> struct F32Tile {
    static constexpr int TJ = BM_ == 64 ? 8 : 4;                  // columns a thread
    static constexpr int WARPS_N = BM_ == 64 ? 2 : 4;             // warps side by side
    static constexpr int STAGE = (BM_ + FBN) * FLD;               // floats
    static constexpr int SMEM = FSTAGES * STAGE * 4;
    static_assert(BM_ * FBN <= FSTAGES * STAGE, "the finished tile reuses the stages");
};

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

template <int BM_>
__global__ void __launch_bounds__(FTHREADS, 2)
gemm_f32_cluster_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                        float* __restrict__ out, int M, int N, int K, long long ldx, long long ldo, int stretches, int w_ready) {
    using T = F32Tile<BM_>;
    constexpr int TJ = T::TJ;
    extern __shared__ __align__(16) float fsm[];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // (tiles in one extent of the grid, column tiles first: the others end at 65,535, which 4.2 million rows exceed)
    const int columns = (N + FBN - 1) / FBN;
    const int m0 = (int)(blockIdx.x / columns) * BM_, n0 = (int)(blockIdx.x % columns) * FBN;
    const int parts = gridDim.z, part = blockIdx.z;               // the cluster spans the whole of z
    const int kt_total = (K + FBK - 1) / FBK;
    const int kt0 = (int)((long long)part * kt_total / parts);
    const int n_kt = (int)((long long)(part + 1) * kt_total / parts) - kt0;
    const int ty = lane >> 3, tx = lane & 7;
    const int wm = (warp / T::WARPS_N) * 32, wn = (warp % T::WARPS_N) * (8 * TJ);

    // A thread copies one 16-byte group (the same columns of k) of every 16th row; the rows' addresses are a step apart.
    // Beyond the matrix nothing is read (the first row's address stands in) and zeros are written.
    const int cr = tid >> 3, cc = (tid & 7) * 4;
    const float* wp = w + (size_t)(n0 + min(cr, N - 1 - n0)) * K + kt0 * FBK + cc;
    const float* xp = x + (size_t)(m0 + min(cr, M - 1 - m0)) * ldx + kt0 * FBK + cc;
    const long long w_step = 16ll * K, x_step = 16ll * ldx;
    const int w_left = N - n0 - cr, x_left = M - m0 - cr;         // rows from this thread's first to the matrix's end
    int k_left = K - kt0 * FBK - cc;                              // the same for k, at the tile that is requested next
    const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(fsm + cr * FLD + cc);
    auto copy = [](uint32_t dst, const float* src, bool in) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    };
    auto fetch_w = [&](int stage, int ahead) {                    // `ahead`: k tiles beyond the one the pointers stand at
        const uint32_t d = dst0 + (stage * T::STAGE + BM_ * FLD) * 4;
        const bool k_in = ahead * FBK < k_left;
        const float* base = k_in ? wp + ahead * FBK : w;
#pragma unroll
        for (int u = 0; u < FBN / 16; ++u) {
            const bool in = k_in && u * 16 < w_left;
            copy(d + u * 16 * FLD * 4, in ? base + u * w_step : w, in);
        }
    };
    auto fetch_x = [&](int stage, int ahead) {
        const uint32_t d = dst0 + stage * T::STAGE * 4;
        const bool k_in = ahead * FBK < k_left;
        const float* base = k_in ? xp + ahead * FBK : x;
#pragma unroll
        for (int u = 0; u < BM_ / 16; ++u) {
            const bool in = k_in && u * 16 < x_left;
            copy(d + u * 16 * FLD * 4, in ? base + u * x_step : x, in);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    if (!w_ready) pdl_wait();                                     // (else the weight does not depend on the kernel before this one)
#pragma unroll
    for (int kt = 0; kt < FSTAGES - 1; ++kt)
        if (kt < n_kt) fetch_w(kt, kt);
    pdl_wait();
#pragma unroll
    for (int kt = 0; kt < FSTAGES - 1; ++kt) {
        if (kt < n_kt) fetch_x(kt, kt);
        commit();                                                 // group 0 also holds every weight tile requested above
    }
    unsigned long long acc[8][TJ];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) acc[i][j] = 0ull;
    wp += (FSTAGES - 1) * FBK; xp += (FSTAGES - 1) * FBK; k_left -= (FSTAGES - 1) * FBK;
    int use = 0, refill = FSTAGES - 1;                            // stages
    const int mine = stretches / parts;                           // stretches of this block: a power of two
    float4 waiting[3 * 2 * TJ];                                   // finished subtrees of 1, 2 and 4 stretches
    int local = 0;
    asm volatile("" : "+r"(local));                               // (an index the compiler cannot see keeps them out of the registers)
    // The sums of the stretch that just ended with the subtrees that waited for them, 2^levels stretches in all: every load of a
    // level in flight together, in the registers of the accumulators' other halves.
    float v[8][TJ];
    auto join = [&](int levels) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TJ; ++j)
                v[i][j] = __uint_as_float((unsigned)acc[i][j]) + __uint_as_float((unsigned)(acc[i][j] >> 32));
#pragma unroll 1
        for (int l = 0; l < levels; ++l) {
            const float4* from = waiting + local + l * 2 * TJ;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TJ; j += 4) {
                    const float4 f = from[(i * TJ + j) / 4];
                    v[i][j] = f.x + v[i][j]; v[i][j + 1] = f.y + v[i][j + 1];
                    v[i][j + 2] = f.z + v[i][j + 2]; v[i][j + 3] = f.w + v[i][j + 3];
                }
        }
    };
    int kt = 0;
    for (int st = 0; ; ++st) {
        const int kt_end = (int)((long long)(part * mine + st + 1) * kt_total / stretches) - kt0;
        for (; kt < kt_end; ++kt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
            __syncthreads();          // tile kt is here, and nobody reads the stage that is refilled next any more
            if (kt + FSTAGES - 1 < n_kt) {
                fetch_w(refill, 0);
                fetch_x(refill, 0);
                wp += FBK; xp += FBK; k_left -= FBK;
            }
            commit();                                                 // an empty group at the end keeps the count
            const float* xs = fsm + use * T::STAGE + (wm + ty) * FLD;
            const float* ws = fsm + use * T::STAGE + (BM_ + wn + tx) * FLD;
            use = use + 1 == FSTAGES ? 0 : use + 1;
            refill = refill + 1 == FSTAGES ? 0 : refill + 1;
#pragma unroll
            for (int c = 0; c < FBK; c += 4) {
                ulonglong2 a[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * 4 * FLD + c);
#pragma unroll
                for (int j = 0; j < TJ; ++j) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * 8 * FLD + c);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[i][j] = fma2(a[i].x, b.x, acc[i][j]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[i][j] = fma2(a[i].y, b.y, acc[i][j]);
                }
            }
        }
        if (st == mine - 1) break;
        const int level = __ffs(~st) - 1;                         // one subtree waits for every trailing one of st
        join(level);
        float4* to = waiting + local + level * 2 * TJ;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < TJ; ++j) {
                if (j % 4 == 0) to[(i * TJ + j) / 4] = make_float4(v[i][j], v[i][j + 1], v[i][j + 2], v[i][j + 3]);
                acc[i][j] = 0ull;
            }
    }
    // the finished part goes to this block's shared memory, row by row ...
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    join(__ffs(mine) - 1);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) fsm[(wm + ty + 4 * i) * FBN + wn + tx + 8 * j] = v[i][j];
    // ... and every block adds and writes its share of the tile, four columns at a time
    if (parts > 1) { sm100::cluster_arrive(); sm100::cluster_wait(); }
    else __syncthreads();
    const bool vec = (((uintptr_t)out | ((uintptr_t)ldo * 4)) & 15) == 0;
    for (int g = part * FTHREADS + tid; g < BM_ * FBN / 4; g += parts * FTHREADS) {
        const int r = g / (FBN / 4), c = (g % (FBN / 4)) * 4;
        const int m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        float v[4];
        if (parts > 1) {
            const uint32_t here = (uint32_t)__cvta_generic_to_shared(fsm + g * 4);
            auto of_block = [&](int z) {
                float4 p;
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w) : "r"(sm100::map_to_cta(here, z)) : "memory");
                return p;
            };
            auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
            float4 sum = add(of_block(0), of_block(1));           // the rest of the tree, over the blocks
            if (parts > 2) sum = add(sum, add(of_block(2), of_block(3)));
            if (parts > 4) sum = add(sum, add(add(of_block(4), of_block(5)), add(of_block(6), of_block(7))));
            v[0] = sum.x; v[1] = sum.y; v[2] = sum.z; v[3] = sum.w;
        } else {
            const float4 p = *reinterpret_cast<const float4*>(fsm + g * 4);
            v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
        }
        float* o = out + (size_t)m * ldo + n;
        if (bias != nullptr) {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] += n + i < N ? bias[n + i] : 0.f;
        }
        if (vec && n + 4 <= N) {
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n + i < N) o[i] = v[i];
        }
    }
    __syncwarp();
    if (parts > 1) { sm100::cluster_arrive(); sm100::cluster_wait(); }       // nobody leaves while its part may still be read
}

// Into how many stretches k is cut, by the weight alone, each of at least four k tiles (128 k): as many parts as pay where the
// step's rows are one row of tiles and the weight's column tiles leave the device idle.  61 rows, in 1, 2, 4 and 8 parts:
// 4,096 x 2,048 124, 84, 59, 34 us; 8,192 x 2,048 125, 106, 62, 66; 12,288 x 2,048 159, 118, 90, 98; 24,576 x 4,096 433, 325, 325, 333;
// 151,936 x 1,024 469, 466, 510, 572.  A finer cut than the parts costs little: 8,192 x 2,048 and 1,000 rows in one part 725 us with
// one stretch, 736 with four, 750 with eight.
int f32_stretches(int N, int k_tiles) {
    const int columns = (N + FBN - 1) / FBN;
    int most = columns <= 33 ? 8 : (columns <= 148 ? 4 : (columns <= 296 ? 2 : 1));
    while (most > 1 && k_tiles / most < 4) most /= 2;
    return most;
}

// Over how many blocks the stretches are dealt out: the cheapest of 1, 2, 4, 8, by rounds of resident clusters times a part's k
// tiles.  clusters[p] is asked of the driver: 296, 148, 71 and 33 on a B200, two blocks a multiprocessor.  A last round that leaves half of
// the places empty takes 0.6 of a full one, since its blocks have a multiprocessor each; clusters of eight are packed and come
// closer to their share.  At K = 2,048 in 1, 2, 4 and 8 parts: 2,048 x 2,048 and 2,048 rows (1.7, 3.5, 7.2, 15.5 rounds) 436, 384, 414,
// 448 us; 2,048 x 2,048 and 320 rows 153, 117, 89, 82; 4,096 x 2,048 and 181 rows 142, 117, 90, 97.
int f32_parts(long long tiles, int k_tiles, int stretches, const int* clusters) {
    int best = 1;
    long long best_cost = -1;
    for (int p = 1; p <= stretches; p *= 2) {
        const long long places = clusters[p];
        if (places < 1) continue;
        const long long rest = tiles % places;
        long long rounds = 10 * (tiles / places);                 // in tenths
        if (rest > 0) rounds += p < 8 ? (2 * rest <= places ? 6 : 10) : std::min(10ll, 3 + 10 * rest / places);
        const long long cost = rounds * (4 * ((k_tiles + p - 1) / p) + 4 + p / 8);
        if (best_cost < 0 || cost < best_cost) { best = p; best_cost = cost; }
    }
    return best;
}

template <int BM_>
int launch_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, long long ldx, long long ldo,
               int w_ready, cudaStream_t s) {
    // the kernel's shared-memory allowance and how many clusters of 1, 2, 4 and 8 blocks run at once, once a device
    struct Facts { int clusters[9]; };
    static PerDevice<Facts> known;
    const Facts* facts = nullptr;
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return (int)e;
    const int error = known.get(dev, &facts, [](Facts& f) {
        auto k = gemm_f32_cluster_kernel<BM_>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Tile<BM_>::SMEM);
        for (int p = 1; p <= 8 && e == cudaSuccess; p *= 2) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(8, 1, p);
            cfg.blockDim = dim3(FTHREADS);
            cfg.dynamicSmemBytes = F32Tile<BM_>::SMEM;
            cudaLaunchAttribute a[1];
            a[0].id = cudaLaunchAttributeClusterDimension;
            a[0].val.clusterDim.x = 1;
            a[0].val.clusterDim.y = 1;
            a[0].val.clusterDim.z = p;
            cfg.attrs = a;
            cfg.numAttrs = 1;
            e = cudaOccupancyMaxActiveClusters(&f.clusters[p], k, &cfg);
        }
        return (int)e;
    });
    if (error) return error;
    const long long tiles = (long long)((N + FBN - 1) / FBN) * ((M + BM_ - 1) / BM_);
    const int k_tiles = (K + FBK - 1) / FBK;
    const int stretches = f32_stretches(N, k_tiles), parts = f32_parts(tiles, k_tiles, stretches, facts->clusters);
    if (tiles > 0x7fffffffll) return RB_ERR_BAD_SIZE;
    dim3 grid((unsigned)tiles, 1, parts);
    cudaError_t e = parts > 1 ? launch_clustered(gemm_f32_cluster_kernel<BM_>, grid, dim3(FTHREADS), dim3(1, 1, parts), F32Tile<BM_>::SMEM, s,
                                                 x, w, bias, out, M, N, K, ldx, ldo, stretches, w_ready)
                              : rb::launch(gemm_f32_cluster_kernel<BM_>, grid, dim3(FTHREADS), F32Tile<BM_>::SMEM, s, x, w, bias, out, M, N,
                                           K, ldx, ldo, stretches, w_ready);
    if (e != cudaSuccess) return (int)e;
    RB_LAUNCH_CHECK();
    return RB_OK;
}

// ---- few rows, 32-bit: one pass over the weight ----------------------------------------------------
constexpr int ROWS_PER_BLOCK = 16;   // weight rows a block: 4 warps of 4 rows (up to 8 step rows) or 8 warps of 2

__device__ __forceinline__ float4 ld_stream(const float* p) {      // read once: do not keep it in the L1
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// A block owns 16 weight rows.  k is walked in tiles of KT: the step's rows of a tile are brought
// into shared memory once for the whole block (two buffers, so that the next tile's copy and the next
// tile's weight loads are in flight while this tile is multiplied), and every lane takes the 16-byte
// groups lane, lane + 32, ... of the tile.  A 16-byte group of a step row read from shared memory
// feeds 4 * ROWS_NW multiply-adds: with 4 weight rows a warp the shared-memory reads no longer bound
// the kernel (with 2 they did, at about half the memory's bandwidth).
template <int MT>
__global__ void __launch_bounds__(MT <= 8 ? 128 : 256)
gemm_rows_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ out, int M, int N, int K, long long ldx, long long ldo, int k_per_split,
                     long long split_stride, int w_ready) {
    constexpr int ROWS_NW = MT <= 8 ? 4 : 2;     // weight rows a warp
    constexpr int ROWS_WARPS = ROWS_PER_BLOCK / ROWS_NW;
    constexpr int KT = 256;                      // floats of k a tile
    constexpr int U = KT / 128;                  // 16-byte groups a lane takes of a tile, per row
    __shared__ __align__(16) float xs[2][MT][KT];
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (blockIdx.x * ROWS_WARPS + warp) * ROWS_NW;
    // blockIdx.y: this block's part of k (a multiple of KT long); its sums go to a partial result of their own,
    // which the consumer adds in order (a narrow weight alone has too few rows to keep the memory busy)
    const int k_lo = blockIdx.y * k_per_split;
    const int k_end = min(K, k_lo + k_per_split);
    out += (size_t)blockIdx.y * split_stride;
    const float* wr[ROWS_NW];
#pragma unroll
    for (int j = 0; j < ROWS_NW; ++j) wr[j] = w + (size_t)min(n0 + j, N - 1) * K;
    float acc[ROWS_NW][MT];
#pragma unroll
    for (int j = 0; j < ROWS_NW; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[j][m] = 0.f;
    auto load_w = [&](float4 (&dst)[U][ROWS_NW], int k0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * 128 + lane * 4;
#pragma unroll
            for (int j = 0; j < ROWS_NW; ++j) dst[u][j] = k < k_end ? ld_stream(wr[j] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // The whole block copies the tile's rows (beyond K or M: zeros), asynchronously: a load that the thread
    // itself had to store would hold it for a round trip to the L2 cache before every tile's arithmetic.
    auto load_x = [&](int buf, int k0) {
        for (int i = threadIdx.x; i < MT * (KT / 4); i += ROWS_WARPS * 32) {
            const int m = i / (KT / 4), k = k0 + (i % (KT / 4)) * 4;
            const bool in = m < M && k < k_end;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&xs[buf][m][(i % (KT / 4)) * 4]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? x + (size_t)m * ldx + k : x),
                         "r"(in ? 16 : 0) : "memory");          // 0 bytes read: the 16 bytes are zero-filled
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // weights that do not depend on the kernel before this one: their first tile is requested at once
    if (!w_ready) pdl_wait();
    float4 wv[U][ROWS_NW];
    load_w(wv, k_lo);
    pdl_wait();
    load_x(0, k_lo);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int buf = 0;
    for (int k0 = k_lo; k0 < k_end; k0 += KT, buf ^= 1) {
        float4 nx[U][ROWS_NW];
        load_w(nx, k0 + KT);
        if (k0 + KT < k_end) load_x(buf ^ 1, k0 + KT);
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 xv = *reinterpret_cast<const float4*>(&xs[buf][m][u * 128 + lane * 4]);
#pragma unroll
                for (int j = 0; j < ROWS_NW; ++j) {
                    acc[j][m] = fmaf(xv.x, wv[u][j].x, acc[j][m]);
                    acc[j][m] = fmaf(xv.y, wv[u][j].y, acc[j][m]);
                    acc[j][m] = fmaf(xv.z, wv[u][j].z, acc[j][m]);
                    acc[j][m] = fmaf(xv.w, wv[u][j].w, acc[j][m]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < ROWS_NW; ++j) wv[u][j] = nx[u][j];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();      // the next tile's rows are in place, and nobody reads this tile's any more
    }
#pragma unroll
    for (int j = 0; j < ROWS_NW; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float v = warp_sum(acc[j][m]);
            if (lane == 0 && m < M && n0 + j < N) out[(size_t)m * ldo + n0 + j] = v + (bias && blockIdx.y == 0 ? bias[n0 + j] : 0.f);
        }
}

template <int MT>
int launch_rows(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, long long ldx,
                long long ldo, int splits, long long split_stride, int w_ready, cudaStream_t s) {
    const int k_per_split = ((K + splits - 1) / splits + 255) / 256 * 256;       // a multiple of the kernel's k tile
    // (a part that lies wholly beyond K, which the rounding to tiles can leave, is written as zeros)
    RB_LAUNCH((gemm_rows_f32_kernel<MT>), dim3((N + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK, splits), dim3(MT <= 8 ? 128 : 256), 0, s,
              x, w, bias, out, M, N, K, ldx, ldo, k_per_split, split_stride, w_ready);
    RB_LAUNCH_CHECK();
    return RB_OK;
}

template <typename XT, typename WT, typename OT>
int launch(const void* x, const void* w, const void* bias, void* out, int M, int N, int K, long long ldx,
           long long ldo, cudaStream_t s) {
    if (M > 64 && N > 64) {       // enough rows and columns to fill the large tiles
        dim3 big((N + LBN - 1) / LBN, (M + LBM - 1) / LBM);
        if (big.y > 65535) return RB_ERR_BAD_SIZE;
        RB_LAUNCH((gemm_tn_large_kernel<XT, WT, OT>), dim3(big), dim3(256), 0, s, (const XT*)x, (const WT*)w, (const float*)bias,
                  (OT*)out, M, N, K, ldx, ldo);
        RB_LAUNCH_CHECK();
        return RB_OK;
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return RB_ERR_BAD_SIZE;
    RB_LAUNCH((gemm_tn_kernel<XT, WT, OT>), dim3(grid), dim3(256), 0, s, (const XT*)x, (const WT*)w, (const float*)bias, (OT*)out, M,
                                                    N, K, ldx, ldo);
    RB_LAUNCH_CHECK();
    return RB_OK;
}
}  // namespace

// How the 32-bit product of more than 16 rows of M x N x K would be cut: into how many stretches of k, over how many blocks, with
// clusters[p] clusters of p blocks resident at once.  Nothing is launched; for tests and tuning.
extern "C" int rb_gemm_f32_plan(int M, int N, int K, const int* clusters, int* stretches, int* parts) {
    const int bm = M <= 32 ? 32 : 64, k_tiles = (K + FBK - 1) / FBK;
    *stretches = f32_stretches(N, k_tiles);
    *parts = f32_parts((long long)((N + FBN - 1) / FBN) * ((M + bm - 1) / bm), k_tiles, *stretches, clusters);
    return RB_OK;
}

// w_ready != 0: w is not written by kernels that this one follows in the stream, so that its first tiles may be read before
// they have ended.
extern "C" int rb_gemm_generic(const void* x, int x_dtype, const void* w, int w_dtype, const void* bias,
                               void* out, int out_dtype, int M, int N, int K, long long ldx, long long ldo,
                               int splits, long long split_stride, int w_ready, void* stream) {
    if (M <= 0 || N <= 0) return RB_OK;
    if (K <= 0 || splits < 1) return RB_ERR_BAD_SIZE;
    // splits > 1: float32 partial sums over parts of k at out + z * split_stride (bias in part 0), for the 32-bit
    // product of at most 16 rows only
    if (splits > 1 && !(x_dtype == RB_F32 && w_dtype == RB_F32 && out_dtype == RB_F32 && M <= 16 && K % 4 == 0 &&
                        ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0))
        return RB_ERR_BAD_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
#define RB_G(XT, WT, OT) return launch<XT, WT, OT>(x, w, bias, out, M, N, K, ldx, ldo, s)
    if (x_dtype == RB_F32 && w_dtype == RB_F32 && out_dtype == RB_F32) {
        // few rows: one pass over the weight (16-byte loads need k, the rows' stride and the pointers to fit)
        if (M <= 16 && K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
            const float *xf = (const float*)x, *wf = (const float*)w, *bf32 = (const float*)bias;
            float* of = (float*)out;
            if (M <= 1) return launch_rows<1>(xf, wf, bf32, of, M, N, K, ldx, ldo, splits, split_stride, w_ready, s);
            if (M <= 2) return launch_rows<2>(xf, wf, bf32, of, M, N, K, ldx, ldo, splits, split_stride, w_ready, s);
            if (M <= 4) return launch_rows<4>(xf, wf, bf32, of, M, N, K, ldx, ldo, splits, split_stride, w_ready, s);
            if (M <= 8) return launch_rows<8>(xf, wf, bf32, of, M, N, K, ldx, ldo, splits, split_stride, w_ready, s);
            return launch_rows<16>(xf, wf, bf32, of, M, N, K, ldx, ldo, splits, split_stride, w_ready, s);
        }
        // more rows, and enough columns to fill a tile's (the same loads); 32 rows a tile while they hold all of them
        if (M > 16 && N > 64 && K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0)
            return M <= 32 ? launch_f32<32>((const float*)x, (const float*)w, (const float*)bias, (float*)out, M, N, K, ldx, ldo, w_ready, s)
                           : launch_f32<64>((const float*)x, (const float*)w, (const float*)bias, (float*)out, M, N, K, ldx, ldo, w_ready, s);
        RB_G(float, float, float);
    }
    if (x_dtype == RB_F32 && w_dtype == RB_BF16 && out_dtype == RB_F32) RB_G(float, bf, float);
    if (x_dtype == RB_BF16 && w_dtype == RB_BF16 && out_dtype == RB_BF16) RB_G(bf, bf, bf);
    if (x_dtype == RB_BF16 && w_dtype == RB_BF16 && out_dtype == RB_F32) RB_G(bf, bf, float);
    if (x_dtype == RB_BF16 && w_dtype == RB_F32 && out_dtype == RB_BF16) RB_G(bf, float, bf);
    if (x_dtype == RB_BF16 && w_dtype == RB_F32 && out_dtype == RB_F32) RB_G(bf, float, float);
#undef RB_G
    return RB_ERR_BAD_DTYPE;
}
