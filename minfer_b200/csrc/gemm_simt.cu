// Plain matrix product on the FP32 pipe: C[M][N] (+)= A[M][K] * W[N][K]^T + bias[N].
//
// This is the true 32-bit path of every projection (FFMA only, no tensor-core mode, so no
// TF32 or bfloat16 staging) and the twin that the tensor-core kernels are checked against.
// Weights are [out][in] row-major and activations token-major as in the reference
// (src/graph/ops.rs:132-136; out[t*od+o] = dot(w[o], x[t]) + bias[o],
// src/graph/cpu_backend.rs:214-247).
//
// Each output element is summed over k in ascending order by one thread; from K = 2,048 on four
// stretches of k are, and their sums are added in order (`f32_stretch`, a function of K only).  Neither M
// nor the place of a row in the batch matters, so a token's result never depends on its neighbours.
// All three kernels below keep that order, so they give the same bits:
//   gemm_f32_few_kernel    up to 16 rows, float32 operands on 16-byte rows
//   gemm_f32_tile_kernel   more rows, the same operands
//   gemm_simt_kernel       everything else (bfloat16 on either side, rows off 16 bytes)
#include "common.cuh"

// k of a stretch: K itself, or a quarter of it in whole 128s (always four stretches).  A product of few
// columns and a long K has too few tiles for the SMs while one thread walks all of K; as a cluster of four
// CTAs a tile it does not.
__host__ __device__ constexpr int f32_stretch(int K) { return K < 2048 ? K : ((K + 511) / 512) * 128; }
#define F32_STRETCHES 4
// how gemm_f32_tile_kernel goes through k: K as one stretch; a cluster of four CTAs a tile, a stretch each;
// one CTA a tile, the four stretches one after the other
#define F32_WHOLE 0
#define F32_SPLIT 1
#define F32_WALK 2

#define BM 64
#define BN 64
#define BK 16

// accumulate: 0  C = acc + bias        1  C = C + acc + bias  (C float32: residual stream)
template <typename TA, typename TW, typename TC, bool LONG>
__global__ void __launch_bounds__(256, 4)
gemm_simt_kernel(const TA* A, const TW* __restrict__ W, const float* __restrict__ bias,
                 TC* C, int M, int N, int K, long long lda, long long ldw,
                 long long ldc, int accumulate) {
    pdl_prologue();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float4 done[LONG ? 4 * 256 : 1];      // every thread's sums of the stretches before this one
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    // LONG (four stretches of k): the sums put away in shared memory, so that four CTAs share an SM as they do for
    // one stretch: in registers, and in kernels of any K, 385 x 3,028 x 10,600 (bfloat16 x float32) took 4,030 us
    // instead of 2,340, 64 x 896 x 4,864 497 instead of 465.  Now, with two tiles of k a round, 1,760 and 411.
    const int stretch = LONG ? f32_stretch(K) : K;
    for (int k0 = 0; k0 < K;) {
        if (LONG && k0 > 0) {
            float4* d = done + tid;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
                if (k0 > stretch) {
                    const float4 o = d[i * 256];
                    v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w;
                }
                d[i * 256] = v;
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
            }
        }
#pragma unroll 2
        for (const int end = LONG ? min(k0 + stretch, K) : K; k0 < end; k0 += BK) {
            // 64 rows x 16 k per operand = 1024 elements, 4 per thread; k fastest for coalescing
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = tid + e * 256;
                const int r = idx >> 4, kk = idx & 15;
                const int k = k0 + kk;
                float a = 0.0f, w = 0.0f;
                if (k < K) {
                    if (m0 + r < M) a = to_f32(A[(size_t)(m0 + r) * lda + k]);
                    if (n0 + r < N) w = to_f32(W[(size_t)(n0 + r) * ldw + k]);
                }
                As[kk][r] = a;
                Ws[kk][r] = w;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[4], w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
        if (LONG) {
            const float4 o = done[i * 256 + tid];
            acc[i][0] = o.x + acc[i][0]; acc[i][1] = o.y + acc[i][1];
            acc[i][2] = o.z + acc[i][2]; acc[i][3] = o.w + acc[i][3];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            TC* c = C + (size_t)m * ldc + n;
            if (accumulate) v += to_f32(*c);
            *c = from_f32<TC>(v);
        }
    }
}

// ---- float32 operands, many rows -------------------------------------------------------------
// Bound by the FP32 pipe (128 multiply-adds a clock and SM).  A thread owns TM x TN outputs in
// float4 groups, so that a step of k costs it (TM + TN) / 4 shared loads for TM * TN multiply-adds.
// Two columns are one packed multiply-add (fma.rn.f32x2: two IEEE results, half the instructions to
// issue).  Tiles lie in shared memory by k (a warp reads 4 rows x 8 column groups), the columns of a
// k swizzled by its quarter so that the transposing stores do not conflict; the next tile's loads are
// in flight in registers while this one is multiplied.
// Measured (us back to back, the tile that is chosen and the 64 x 64 x 16 kernel above in brackets):
// 385 x 9,728 x 896 192 (64 x 64) [387], 385 x 151,936 x 896 2,546 (128 x 128) [5,617]; of a K in stretches, with
// K as one in front: 385 x 896 x 4,864 227 -> 129 (32 x 64, a cluster a tile), 64 x 896 x 4,864 93 -> 56 (the same),
// 1,600 x 2,048 x 8,448 1,380 -> 1,212 (128 x 128, the same), 1,600 x 8,448 x 2,048 1,082 -> 1,095 (128 x 128, one CTA a
// tile) = 51 TFLOP/s of the pipe's 74; as a cluster a tile that took 1,197, 634 x 6,420 x 2,080 481 instead of 390.
// Plain multiply-adds instead of packed ones: 2 to 7 % slower.  AHEAD 2 (loads two tiles ahead) for the smallest tile,
// whose product of a tile is shorter than a trip to memory: 64 x 896 x 4,864 129 -> 95; for 64 x 64 it lost (240 -> 280).
__device__ __forceinline__ unsigned long long f32x2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma_f32x2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ float4 f32_sums(unsigned long long a, unsigned long long b) {
    return make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)),
                       __uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

// An operand's 16 bytes, never moved above the wait for the kernel before (as a load through a const
// __restrict__ pointer may be).
__device__ __forceinline__ float4 load16(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// every thread of the cluster's CTAs comes here; writes to shared memory before it are seen after it
__device__ __forceinline__ void cluster_wait_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 load16_of_rank(unsigned smem, int rank) {
    float4 v;
    asm volatile(
        "{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %4, %5;\n"
        " ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n}\n"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem), "r"(rank) : "memory");
    return v;
}

template <int ROWS, int THREADS, int BKT>
__device__ __forceinline__ void f32_tile_fetch(const float* src, long long ld, int row0, int rows,
                                               int k0, int K, float4* held) {
#pragma unroll
    for (int e = 0; e < ROWS * (BKT / 4) / THREADS; ++e) {
        const int idx = (int)threadIdx.x + e * THREADS;
        const int r = row0 + idx / (BKT / 4), k = k0 + (idx % (BKT / 4)) * 4;
        held[e] = (r < rows && k < K) ? load16(src + (size_t)r * ld + k)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
template <int ROWS, int THREADS, int BKT>
__device__ __forceinline__ void f32_tile_put(float (*tile)[ROWS], const float4* held) {
#pragma unroll
    for (int e = 0; e < ROWS * (BKT / 4) / THREADS; ++e) {
        const int idx = (int)threadIdx.x + e * THREADS;
        const int q = idx % (BKT / 4), c = (idx / (BKT / 4)) ^ (q * (128 / BKT));
        tile[q * 4 + 0][c] = held[e].x;
        tile[q * 4 + 1][c] = held[e].y;
        tile[q * 4 + 2][c] = held[e].z;
        tile[q * 4 + 3][c] = held[e].w;
    }
}

// a warp covers 4 TM rows x 8 TN columns
template <int BM_, int BN_, int TM, int TN>
struct F32Tile {
    static constexpr int WARPS_N = BN_ / (8 * TN);
    static constexpr int THREADS = 32 * WARPS_N * (BM_ / (4 * TM));
};

// F32_SPLIT: a cluster of four CTAs has a tile, CTA r the stretch r of k; they add their sums in order of the
// stretches through distributed shared memory, each a quarter of the tile's rows.  F32_WALK: a CTA has a tile and
// puts every thread's sums away in shared memory behind a stretch.
template <int BM_, int BN_, int TM, int TN, int BKT, int AHEAD, int FORM>
__global__ void __launch_bounds__(F32Tile<BM_, BN_, TM, TN>::THREADS,
                                  (AHEAD == 1 ? 512 : 384) / F32Tile<BM_, BN_, TM, TN>::THREADS)
gemm_f32_tile_kernel(const float* A, const float* W, const float* __restrict__ bias, float* C,
                     int M, int N, int K_all, long long lda, long long ldw,
                     long long ldc, int accumulate) {
    constexpr int THREADS = F32Tile<BM_, BN_, TM, TN>::THREADS;
    constexpr int WARPS_N = F32Tile<BM_, BN_, TM, TN>::WARPS_N;
    constexpr int FA = BM_ * (BKT / 4) / THREADS, FW = BN_ * (BKT / 4) / THREADS;
    constexpr bool SPLIT = FORM == F32_SPLIT, WALK = FORM == F32_WALK;
    __shared__ __align__(16) float pool[2 * BKT * (BM_ + BN_)];
    extern __shared__ __align__(16) float f32_done[];  // WALK: every thread's sums of the stretches before
    float (*As)[BKT][BM_] = reinterpret_cast<float (*)[BKT][BM_]>(pool);
    float (*Ws)[BKT][BN_] = reinterpret_cast<float (*)[BKT][BN_]>(pool + 2 * BKT * BM_);
    const int k_first = SPLIT ? (int)blockIdx.z * f32_stretch(K_all) : 0;
    const int K = SPLIT ? min(K_all, k_first + f32_stretch(K_all)) : K_all;       // this CTA's end
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ty = (warp / WARPS_N) * 4 * TM + (lane >> 3) * 4;     // + 16 per group of 4 rows
    const int tx = (warp % WARPS_N) * 8 * TN + (lane & 7) * 4;      // + 32 per group of 4 columns
    // row tiles run fastest: CTAs side by side read the same weights
    const int m0 = blockIdx.x * BM_, n0 = blockIdx.y * BN_;
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    pdl_prologue();
    float4 ha[AHEAD][FA], hw[AHEAD][FW];              // the next AHEAD tiles, on their way
    auto fetch = [&](int t, int set) {
        f32_tile_fetch<BM_, THREADS, BKT>(A, lda, m0, M, k_first + t * BKT, K, ha[set]);
        f32_tile_fetch<BN_, THREADS, BKT>(W, ldw, n0, N, k_first + t * BKT, K, hw[set]);
    };
    auto put = [&](int t, int set) {
        f32_tile_put<BM_, THREADS, BKT>(As[t & 1], ha[set]);
        f32_tile_put<BN_, THREADS, BKT>(Ws[t & 1], hw[set]);
    };
    auto multiply = [&](int t) {
        const float (*at)[BM_] = As[t & 1];
        const float (*wt)[BN_] = Ws[t & 1];
#pragma unroll
        for (int kk = 0; kk < BKT; ++kk) {
            const int swz = (kk >> 2) * (128 / BKT);
            float4 w[TN / 4];
#pragma unroll
            for (int h = 0; h < TN / 4; ++h)
                w[h] = *reinterpret_cast<const float4*>(&wt[kk][(tx + h * 32) ^ swz]);
#pragma unroll
            for (int g = 0; g < TM / 4; ++g) {
                const float4 a4 = *reinterpret_cast<const float4*>(&at[kk][(ty + g * 16) ^ swz]);
                const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const unsigned long long aa = f32x2(a[i], a[i]);
#pragma unroll
                    for (int h = 0; h < TN / 4; ++h) {
                        fma_f32x2(acc[g * 4 + i][h * 2], aa, f32x2(w[h].x, w[h].y));
                        fma_f32x2(acc[g * 4 + i][h * 2 + 1], aa, f32x2(w[h].z, w[h].w));
                    }
                }
            }
        }
    };
    // tiles beyond the last are fetched as zeros (no load) and never multiplied
    const int tiles = (K - k_first + BKT - 1) / BKT;
    fetch(0, 0);
    put(0, 0);
    if (AHEAD == 2) fetch(1, 1);
    __syncthreads();
    const int per = WALK ? f32_stretch(K_all) / BKT : tiles;         // tiles of a stretch: an even number
    for (int t = 0, end = per; t < tiles; t += AHEAD) {
        if (WALK && t == end) {
            float4* d = reinterpret_cast<float4*>(f32_done) + threadIdx.x;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int h = 0; h < TN / 4; ++h) {
                    float4 v = f32_sums(acc[i][h * 2], acc[i][h * 2 + 1]);
                    float4& at = d[(i * (TN / 4) + h) * THREADS];
                    if (t > per) { const float4 o = at; v.x = o.x + v.x; v.y = o.y + v.y; v.z = o.z + v.z; v.w = o.w + v.w; }
                    at = v;
                    acc[i][h * 2] = acc[i][h * 2 + 1] = 0ull;
                }
            end += per;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            if (t + u >= tiles) break;
            fetch(t + u + AHEAD, u);                  // (set u was put into shared memory a tile ago)
            multiply(t + u);
            put(t + u + 1, (u + 1) % AHEAD);
            __syncthreads();
        }
    }
    if (SPLIT) {
        // a group of columns at a time: BM_ rows x COLS sums of every CTA, its own in `pool`
        constexpr int COLS = 32 * WARPS_N, QUADS = COLS / 4, MINE = BM_ / F32_STRETCHES;
        static_assert(BM_ * COLS <= 2 * BKT * (BM_ + BN_), "a group of columns fits the tiles' memory");
        const int own = (int)blockIdx.z * MINE;
#pragma unroll
        for (int h = 0; h < TN / 4; ++h) {
            if (h > 0) cluster_wait_all();                            // the group before has been read
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                *reinterpret_cast<float4*>(pool + (ty + (i >> 2) * 16 + (i & 3)) * COLS +
                                           (warp % WARPS_N) * 32 + (lane & 7) * 4) =
                    f32_sums(acc[i][h * 2], acc[i][h * 2 + 1]);
            }
            cluster_wait_all();
            for (int idx = threadIdx.x; idx < MINE * QUADS; idx += THREADS) {
                const int r = own + idx / QUADS, q = idx % QUADS;
                const int m = m0 + r, n = n0 + (q / 8) * 8 * TN + h * 32 + (q % 8) * 4;
                const unsigned at = (unsigned)__cvta_generic_to_shared(pool + r * COLS + q * 4);
                float v[4];
#pragma unroll
                for (int z = 0; z < F32_STRETCHES; ++z) {
                    const float4 p = load16_of_rank(at, z);
                    v[0] = z == 0 ? p.x : v[0] + p.x;
                    v[1] = z == 0 ? p.y : v[1] + p.y;
                    v[2] = z == 0 ? p.z : v[2] + p.z;
                    v[3] = z == 0 ? p.w : v[3] + p.w;
                }
                if (m >= M) continue;
                float* c = C + (size_t)m * ldc + n;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (n + j >= N) break;
                    if (bias != nullptr) v[j] += bias[n + j];
                    if (accumulate) v[j] += c[j];
                }
                if (n + 3 < N && ((((uintptr_t)c) & 15) == 0)) {
                    *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (n + j < N) c[j] = v[j];
                }
            }
        }
        cluster_wait_all();                                           // nobody reads this CTA's sums any more
        return;
    }
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
        const int n = n0 + tx + h * 32;
        float b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = (bias != nullptr && n + j < N) ? bias[n + j] : 0.0f;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + ty + (i >> 2) * 16 + (i & 3);
            if (m >= M) continue;
            float* c = C + (size_t)m * ldc + n;
            const float4 sum = f32_sums(acc[i][h * 2], acc[i][h * 2 + 1]);
            float v[4] = {sum.x, sum.y, sum.z, sum.w};
            if (WALK) {
                const float4 o = reinterpret_cast<const float4*>(f32_done)[(i * (TN / 4) + h) * THREADS + threadIdx.x];
                v[0] = o.x + v[0]; v[1] = o.y + v[1]; v[2] = o.z + v[2]; v[3] = o.w + v[3];
            }
            if (bias != nullptr) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += b[j];
            }
            if (n + 3 < N && ((((uintptr_t)c) & 15) == 0)) {
                if (accumulate) {
                    const float4 o = *reinterpret_cast<const float4*>(c);
                    v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
                }
                *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n + j < N) c[j] = accumulate ? v[j] + c[j] : v[j];
            }
        }
    }
}

// ---- float32 operands, up to 16 rows -----------------------------------------------------------
// Bound by latency: what a step of few tokens waits for is one round trip to memory and a chain of
// K multiply-adds.  A warp owns 8 columns and all rows, a thread RT outputs of one column; the warp
// keeps a ring of k chunks filled by asynchronous copies of its own and waits for no other warp.
// 1 x 896 x 896 88 -> 12 us (a launch's own time), 8 x 896 x 4,864 466 -> 31.
template <int RT> struct F32Few {
    static constexpr int WARPS = 2, STAGES = 2;
    static constexpr int KC = RT == 1 ? 128 : 64, PITCH = KC + 4;    // + 4: 8 columns without conflict
    static constexpr int ROWS = 8 + 4 * RT;                          // weight rows, then activation rows
};

__device__ __forceinline__ void copy16_async(void* smem, const void* src, bool real) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = real ? 16 : 0;                                 // 0: the 16 bytes become zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// LONG: four stretches of k, one behind the other; 8 x 896 x 4,864 29.4 us (29.1 as one chain).  The end of a stretch is
// counted and stands behind the wait for a chunk's copies: with a remainder for every chunk, in kernels of any K, it took
// 36.3 (8 x 896 x 896 7.9 instead of 6.6), with a loop around the stretches 36.8; a quarter of a chunk from each
// stretch, as four independent chains, 29.6, but 8 x 5,228 x 15,960 325 instead of 245: 64-byte pieces of a row.
template <int RT, bool LONG>
__global__ void __launch_bounds__(F32Few<RT>::WARPS * 32)
gemm_f32_few_kernel(const float* A, const float* W, const float* __restrict__ bias, float* C, int M, int N,
                    int K, long long lda, long long ldw, long long ldc, int accumulate) {
    typedef F32Few<RT> T;
    __shared__ __align__(16) float ring[T::WARPS][T::STAGES][T::ROWS][T::PITCH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = ((int)blockIdx.x * T::WARPS + warp) * 8;
    const int col = lane & 7, grp = lane >> 3;
    pdl_prologue();
    if (n0 >= N) return;                                             // no block-wide barrier below
    auto fetch = [&](int chunk) {
        const int k0 = chunk * T::KC;
        float (*st)[T::PITCH] = ring[warp][chunk % T::STAGES];
#pragma unroll
        for (int i = lane; i < T::ROWS * (T::KC / 4); i += 32) {
            const int r = i / (T::KC / 4), k = (i % (T::KC / 4)) * 4;
            const bool weight = r < 8;
            const int row = weight ? n0 + r : r - 8;
            const bool real = k0 + k < K && row < (weight ? N : M);
            const float* src = weight ? W : A;
            if (real) src += (size_t)row * (weight ? ldw : lda) + k0 + k;
            copy16_async(&st[r][k], src, real);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int chunks = (K + T::KC - 1) / T::KC;
    fetch(0);
    float acc[RT], done[RT];                                         // done: the stretches before this one
#pragma unroll
    for (int i = 0; i < RT; ++i) acc[i] = 0.0f;
    const int per = LONG ? f32_stretch(K) / T::KC : chunks;          // chunks of a stretch
    int end = per;
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            fetch(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        if (LONG && c == end) {
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                done[i] = c == per ? acc[i] : done[i] + acc[i];
                acc[i] = 0.0f;
            }
            end += per;
        }
        const float (*st)[T::PITCH] = ring[warp][c % T::STAGES];
        const int ks = min(T::KC, K - c * T::KC);
#pragma unroll 8
        for (int k = 0; k < ks; k += 4) {
            const float4 w = *reinterpret_cast<const float4*>(&st[col][k]);
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(&st[8 + grp + 4 * i][k]);
                acc[i] = fmaf(a.x, w.x, acc[i]);
                acc[i] = fmaf(a.y, w.y, acc[i]);
                acc[i] = fmaf(a.z, w.z, acc[i]);
                acc[i] = fmaf(a.w, w.w, acc[i]);
            }
        }
        __syncwarp();                                                // all lanes are done with this stage
    }
    const int n = n0 + col;
    if (n >= N) return;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int m = grp + 4 * i;
        if (m >= M) continue;
        float v = LONG ? done[i] + acc[i] : acc[i];
        if (bias != nullptr) v += bias[n];
        float* c = C + (size_t)m * ldc + n;
        if (accumulate) v += *c;
        *c = v;
    }
}

template <int BM_, int BN_, int TM, int TN, int BKT, int AHEAD>
static int launch_f32_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                            long long lda, long long ldw, long long ldc, int accumulate, int form,
                            cudaStream_t stream) {
    const dim3 grid((M + BM_ - 1) / BM_, (N + BN_ - 1) / BN_, form == F32_SPLIT ? F32_STRETCHES : 1);
    const dim3 block(F32Tile<BM_, BN_, TM, TN>::THREADS);
    if (form == F32_WHOLE) {
        mf_launch(gemm_f32_tile_kernel<BM_, BN_, TM, TN, BKT, AHEAD, F32_WHOLE>, grid, block, 0, stream, A, W, bias, C,
                  M, N, K, lda, ldw, ldc, accumulate);
        return 0;
    }
    if (form == F32_WALK) {
        constexpr int done = BM_ * BN_ * (int)sizeof(float);
        static bool configured[64] = {false};
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MF_ERR_UNSUPPORTED;
        if (!configured[dev]) {
            cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<BM_, BN_, TM, TN, BKT, AHEAD, F32_WALK>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, done);
            if (e != cudaSuccess) return (int)e;
            configured[dev] = true;
        }
        mf_launch(gemm_f32_tile_kernel<BM_, BN_, TM, TN, BKT, AHEAD, F32_WALK>, grid, block, done, stream, A, W, bias,
                  C, M, N, K, lda, ldw, ldc, accumulate);
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 1;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = F32_STRETCHES;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = mf_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<BM_, BN_, TM, TN, BKT, AHEAD, F32_SPLIT>, A, W, bias, C, M, N, K,
                       lda, ldw, ldc, accumulate);
    return 0;
}

// The tile of a float32 product of more than 16 rows (an index into `tiles`; -1: the general kernel, whose
// grid takes more columns) and how it goes through k: what lets the fullest SM be done first.  `shared`: what a
// CTA takes of a full SM.  `few`: what the product takes when its CTAs are few: launched while the kernel before
// still runs, they pile up on the SMs that are free, as many as one takes (2, 4 and 3 of these tiles).  Both in
// units of the 64 x 64 tile's share, 27 us a thousand k, fitted to products behind a norm, each timed with every
// tile; `cut` the same for a cluster of four CTAs a tile, fitted in the same way to 190 products of 17 to 4,096
// rows and 2,048 to 18,944 k in both forms.
//   K below 2,048, 255 products: the choice is within 0.1 % of the best tile on average (13 % at worst), and
//   within 1.1 % (21 %) of 109 products back to back; 66 others 0.3 % (6 %) and 0.7 % (24 %).
//   From 2,048 on, 190 products: 0.6 % (16 %) behind a norm, 0.9 % (19 %) back to back.  A cluster a tile
//   whatever the size, by the numbers of the other form: 1.7 % (25 %) and 1.9 % (24 %); none is slower than
//   with that by more than 1 %.
// us, 128 x 128 / 64 x 64 / 32 x 64, norm and product: 385 x 9,728 x 896 241 / 194 / 205; clusters, then one CTA
// a tile: 200 x 4,096 x 2,048 107 / 116 / 115, 376 / 223 / 135; 385 x 896 x 4,864 248 / 143 / 132,
// 476 / 273 / 240; 1,600 x 8,448 x 2,048 1,202 / 1,274 / 1,570, 1,099 / 1,242 / 1,476.
struct F32Cut { int tile, form; };
static F32Cut f32_cut(int M, int N, int K, int sms) {
    static const struct { int bm, bn; double few, shared, cut_few, cut_shared; } tiles[] = {
        {128, 128, 6.4, 3.3, 5.92, 3.18}, {64, 64, 3.9, 1.0, 3.73, 0.921}, {32, 64, 1.8, 0.58, 1.65, 0.598}};
    F32Cut best = {-1, F32_WHOLE};
    double least = 0.0;
    const int stretch = f32_stretch(K);
    for (int i = 0; i < 3; ++i) {
        const long long nt = ((long long)N + tiles[i].bn - 1) / tiles[i].bn;
        const long long ctas = ((long long)M + tiles[i].bm - 1) / tiles[i].bm * nt;
        if (nt > 65535) continue;                                    // the grid's second dimension
        const double whole = (double)((ctas + sms - 1) / sms) * tiles[i].shared;
        const double cost = (whole > tiles[i].few ? whole : tiles[i].few) * K;
        if (best.tile < 0 || cost < least) { best = {i, stretch < K ? F32_WALK : F32_WHOLE}; least = cost; }
        if (stretch == K) continue;
        // (49: adding the four parts, in k)
        const double part = (double)((F32_STRETCHES * ctas + sms - 1) / sms) * tiles[i].cut_shared;
        const double cut = (part > tiles[i].cut_few ? part : tiles[i].cut_few) * (stretch + 49);
        if (cut < least) { best = {i, F32_SPLIT}; least = cut; }
    }
    return best;
}
// The tile below 2,048 k.
extern "C" int mf_gemm_f32_tile(int M, int N, int sms) { return f32_cut(M, N, 1024, sms).tile; }
// The tile, and in `form` 0 (K as one stretch), 1 (a cluster a tile) or 2 (one CTA a tile, four stretches).
extern "C" int mf_gemm_f32_cut(int M, int N, int K, int sms, int* form) {
    const F32Cut c = f32_cut(M, N, K, sms);
    *form = c.form;
    return c.tile;
}

// Float32 operands whose rows start on 16 bytes; false: the general kernel has to run.
static bool launch_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                       long long lda, long long ldw, long long ldc, int accumulate, cudaStream_t stream, int* err) {
    if (((uintptr_t)A | (uintptr_t)W) & 15 || (K | lda | ldw) & 3) return false;
    if (M <= 16) {
        const int warps = (int)(((long long)N + 7) / 8);
#define MF_FEW(RT)                                                                                       \
    if (f32_stretch(K) < K)                                                                              \
        mf_launch(gemm_f32_few_kernel<RT, true>, dim3((warps + F32Few<RT>::WARPS - 1) / F32Few<RT>::WARPS), \
                  dim3(F32Few<RT>::WARPS * 32), 0, stream, A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate); \
    else                                                                                                 \
        mf_launch(gemm_f32_few_kernel<RT, false>, dim3((warps + F32Few<RT>::WARPS - 1) / F32Few<RT>::WARPS), \
                  dim3(F32Few<RT>::WARPS * 32), 0, stream, A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate)
        if (M <= 4) { MF_FEW(1); }
        else if (M <= 8) { MF_FEW(2); }
        else { MF_FEW(4); }
#undef MF_FEW
        return true;
    }
    const F32Cut cut = f32_cut(M, N, K, mf_sm_count());
#define MF_TILE(BM_, BN_, TM, TN, BKT, AHEAD)                                                              \
    *err = launch_f32_tile<BM_, BN_, TM, TN, BKT, AHEAD>(A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, \
                                                         cut.form, stream)
    switch (cut.tile) {
        case 0: MF_TILE(128, 128, 8, 8, 16, 1); break;
        case 1: MF_TILE(64, 64, 4, 8, 32, 1); break;
        case 2: MF_TILE(32, 64, 4, 4, 32, 2); break;
        default: return false;
    }
#undef MF_TILE
    return true;
}

extern "C" int mf_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype,
                            const float* bias, void* C, int c_dtype, int M, int N, int K,
                            long long lda, long long ldw, long long ldc, int accumulate,
                            cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return MF_ERR_ARGUMENT;
    if (accumulate && c_dtype != MF_DTYPE_F32) return MF_ERR_UNSUPPORTED;
    int err = 0;
    if (a_dtype == MF_DTYPE_F32 && w_dtype == MF_DTYPE_F32 && c_dtype == MF_DTYPE_F32 &&
        launch_f32((const float*)A, (const float*)W, bias, (float*)C, M, N, K, lda, ldw, ldc, accumulate, stream, &err))
        return err != 0 ? err : MF_LAUNCH_CHECK();
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return MF_ERR_UNSUPPORTED;
#define MF_GEMM(TA, TW, TC)                                                                                   \
    if (f32_stretch(K) < K)                                                                                   \
        mf_launch(gemm_simt_kernel<TA, TW, TC, true>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, \
                  bias, (TC*)C, M, N, K, lda, ldw, ldc, accumulate);                                           \
    else                                                                                                      \
        mf_launch(gemm_simt_kernel<TA, TW, TC, false>, dim3(grid), dim3(256), 0, stream, (const TA*)A, (const TW*)W, \
                  bias, (TC*)C, M, N, K, lda, ldw, ldc, accumulate)
    typedef __nv_bfloat16 bf16;
    const int key = a_dtype * 4 + w_dtype * 2 + c_dtype;
    switch (key) {
        case 0: MF_GEMM(float, float, float); break;
        case 1: MF_GEMM(float, float, bf16); break;
        case 2: MF_GEMM(float, bf16, float); break;
        case 3: MF_GEMM(float, bf16, bf16); break;
        case 4: MF_GEMM(bf16, float, float); break;
        case 5: MF_GEMM(bf16, float, bf16); break;
        case 6: MF_GEMM(bf16, bf16, float); break;
        case 7: MF_GEMM(bf16, bf16, bf16); break;
        default: return MF_ERR_UNSUPPORTED;
    }
#undef MF_GEMM
    return MF_LAUNCH_CHECK();
}
