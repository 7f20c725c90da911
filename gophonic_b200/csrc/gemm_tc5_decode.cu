// Y[M, N] = X[M, K] * W[N, K]^T for 9 to 256 rows on tcgen05: the product of a decode step, or of
// a short prompt, when there are too many rows for the fragment-streaming kernel and too few for
// the tiled kernels to give every SM a share of the weights.  (Also for fewer rows where the
// dispatch rule finds it the faster stream: head-sized outputs, and products long on both sides.)
//
// The weights take the M side of the instruction: a CTA owns 128 rows of W and a slice of K, and
// computes Y^T[128, batch] with UMMA M = 128, N = 16 / 32 / 64 / 128 / 256 (the batch rounded up;
// TMA fills the missing rows of X with zeros).  Per K step of 64 a stage holds 16 KB of W from HBM
// and 2 to 32 KB of X from L2; up to 64 rows four stages deep, above that three; two CTAs to an SM
// (one at 256 columns), so every SM keeps tens of KB of weights in flight.  K is cut into slices so
// that about that many CTAs exist even for narrow outputs.  The CTAs that share a tile (1, 2, 4 or 8
// slices of K) form a thread-block cluster:
// each leaves its partial tile in its own shared memory, and after a cluster barrier each CTA adds
// the slices, in slice order, for its share of the batch rows (a warp a row), reading the other CTAs'
// shared memory directly (distributed shared memory).  No scratch in global memory, and the sum does not
// depend on timing.  With the gate/up rows of a SwiGLU interleaved in blocks of eight the
// activation is applied in the same epilogue.
//
// Up to 64 rows the residual's row-wise work can be folded into the product as in the few-row
// kernel (gemm_skinny_fold.cu).  As producer (epi 2) Y is the fp32 residual: Y += product, one
// thread and one fp32 addition per element; one partial sum of squares per row and tile of 128
// columns goes to stats_out[row][tile]; and the new rows times the next norm's weight go out as
// bfloat16.  As consumer (stats_in given) the activations are such rows and the finished sums are
// multiplied by the rows' norm factors, the partial sums added up in index order.
//
// Roles by warp as in the tiled kernel: warp 0 loads by TMA, warp 1 issues tcgen05.mma, warps
// 2-5 read tensor memory (lane = weight row, column = batch row) and store.  Barrier waits are
// bounded; a wait that gives up is recorded and read with gb_gemm_tc5_decode_status().
#include "api.h"
#include "tc5.cuh"

namespace {

__device__ int g_status;

constexpr int BMW = 128, BK = 64, THREADS = 192;
constexpr int W_BYTES = BMW * BK * 2;
constexpr int MAX_SPLITS = 8;

// the folded variants' extra operands (all null / 0 for the plain product)
struct DecodeFold {
    const float* stats_in;   // [rows][stats_count] partial sums of squares of the rows X was made from
    int stats_count;
    int64_t stats_in_stride;
    float eps;
    int norm_n;              // width of the normed rows
    float* stats_out;        // epi 2: [rows][tiles]
    int64_t stats_out_stride;
    const float* next_w;     // epi 2, optional: weight of the norm that reads the residual next
    __nv_bfloat16* xn_out;   // [rows][N] = bf16(Y * next_w)
    int64_t ldxn;
};
constexpr int FOLD_ROWS = GB_FOLD_MAX_ROWS;

// x / (1 + exp(-x)) without overflow on either side, and without a branch: the lanes of a warp hold values of both signs
__device__ __forceinline__ float silu_f(float x) {
    const float e = expf(-fabsf(x));
    return (x >= 0.f ? x : x * e) / (1.f + e);
}

// Four neighbouring elements of a row, of which the first `have` exist (the others read as zero and are not written); `vec`:
// the row's address allows one access of all four.
__device__ __forceinline__ float4 load4(const float* p, int have, bool vec) {
    if (vec && have >= 4) return *reinterpret_cast<const float4*>(p);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (have > 0) v.x = p[0];
    if (have > 1) v.y = p[1];
    if (have > 2) v.z = p[2];
    if (have > 3) v.w = p[3];
    return v;
}
__device__ __forceinline__ void store4(float* p, const float4& v, int have, bool vec) {
    if (vec && have >= 4) {
        *reinterpret_cast<float4*>(p) = v;
        return;
    }
    if (have > 0) p[0] = v.x;
    if (have > 1) p[1] = v.y;
    if (have > 2) p[2] = v.z;
    if (have > 3) p[3] = v.w;
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float4& v, int have, bool vec) {
    if (vec && have >= 4) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&lo);
        u.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(p) = u;
        return;
    }
    if (have > 0) p[0] = __float2bfloat16_rn(v.x);
    if (have > 1) p[1] = __float2bfloat16_rn(v.y);
    if (have > 2) p[2] = __float2bfloat16_rn(v.z);
    if (have > 3) p[3] = __float2bfloat16_rn(v.w);
}
__device__ __forceinline__ void store2(float* p, float a, float b, bool vec) {
    if (vec) {
        *reinterpret_cast<float2*>(p) = make_float2(a, b);
        return;
    }
    p[0] = a;
    p[1] = b;
}
__device__ __forceinline__ void store2(__nv_bfloat16* p, float a, float b, bool vec) {
    if (vec) {
        *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
        return;
    }
    p[0] = __float2bfloat16_rn(a);
    p[1] = __float2bfloat16_rn(b);
}

// value v of (weight row n, batch row b) -> Y, plain or through the SwiGLU epilogue; `other` is the
// value of weight row n + 8 (the up row of a gate row), fetched by the caller with a shuffle
template <typename TC>
__device__ __forceinline__ void store_out(TC* __restrict__ Y, int64_t ldy, int b, int n, int N, float v, float other, int epi) {
    if (epi == 0) {
        if (n < N) Y[(int64_t)b * ldy + n] = from_f32<TC>(v);
    } else {
        if ((n & 15) < 8 && n + 8 < N) Y[(int64_t)b * ldy + ((n >> 4) << 3) + (n & 7)] = from_f32<TC>(silu_f(v) * other);
    }
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }

// Registers for the CTAs that shared memory lets an SM hold, or a few more where nothing spills: three of 64 columns and four stages
// (99 KB, two an SM) spilled 48 bytes a thread (64 x 2048 x 6144 12.4 us, 11.1 without).
template <typename TC, int NB, int STAGES>  // NB = batch columns of the instruction: 16 to 256; STAGES deep
__global__ void __launch_bounds__(THREADS, NB <= 32 ? 4 : NB == 64 && STAGES >= 4 ? 2 : 3) gemm_tc5_decode_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                 const __grid_constant__ CUtensorMap map_x, TC* __restrict__ Y,
                                                                 int M, int N, int K, int64_t ldy, int splits, int kb_per_split,
                                                                 int epi, int vec, DecodeFold fold) {
    constexpr int X_BYTES = NB * BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    constexpr int TMEM_COLS = NB < 32 ? 32 : NB;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], accum_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_s;
    __shared__ float rs_s[FOLD_ROWS];          // the rows' norm factors (consumer)
    __shared__ float sq_part[4][FOLD_ROWS];    // sums of squares of the four epilogue warps' rows (producer)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BMW, split = blockIdx.y;
    const int KB = (K + BK - 1) / BK;
    const int kb0 = split * kb_per_split;
    const int kb1 = kb0 + kb_per_split < KB ? kb0 + kb_per_split : KB;
    const int KT = kb1 > kb0 ? kb1 - kb0 : 0;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&map_x) : "memory");
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&accum_bar, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    // Barriers and tensor memory were set up while the kernel ahead was still running.  The weights
    // do not depend on that kernel either: the loading thread requests the first stages' weights
    // before it waits, and only their activations after.
    const int early = KT < STAGES ? KT : STAGES;
    if (warp == 0 && lane == 0) {
        for (int kt = 0; kt < early; kt++) {
            mbar_expect_tx(&full_bar[kt], STAGE_BYTES);
            tma_load_2d(tiles + (size_t)kt * STAGE_BYTES, &map_w, (kb0 + kt) * BK, n0, &full_bar[kt]);
        }
    }
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        if (lane == 0) {
            int issued = early;
            for (int kt = 0; kt < early; kt++)
                tma_load_2d(tiles + (size_t)kt * STAGE_BYTES + W_BYTES, &map_x, (kb0 + kt) * BK, 0, &full_bar[kt]);
            for (int kt = early; kt < KT; kt++) {
                const int s = kt % STAGES;
                const uint32_t phase = (uint32_t)(kt / STAGES) & 1u;
                if (!mbar_wait(&empty_bar[s], phase ^ 1u)) {
                    atomicCAS(&g_status, 0, 1);
                    abort_s = 1;
                    break;
                }
                if (*(volatile int*)&abort_s) break;
                mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                unsigned char* st = tiles + (size_t)s * STAGE_BYTES;
                tma_load_2d(st, &map_w, (kb0 + kt) * BK, n0, &full_bar[s]);
                tma_load_2d(st + W_BYTES, &map_x, (kb0 + kt) * BK, 0, &full_bar[s]);
                issued = kt + 1;
            }
            if (*(volatile int*)&abort_s) {
                for (int kt = issued > STAGES ? issued - STAGES : 0; kt < issued; kt++)
                    mbar_wait(&full_bar[kt % STAGES], (uint32_t)(kt / STAGES) & 1u);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = instr_desc(BMW, NB);
            bool ok = true;
            for (int kt = 0; kt < KT; kt++) {
                const int s = kt % STAGES;
                const uint32_t phase = (uint32_t)(kt / STAGES) & 1u;
                if (!mbar_wait(&full_bar[s], phase)) {
                    atomicCAS(&g_status, 0, 2);
                    abort_s = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t w_addr = s32(tiles + (size_t)s * STAGE_BYTES);
                const uint64_t adesc = smem_desc(w_addr), bdesc = smem_desc(w_addr + W_BYTES);
#pragma unroll
                for (int k = 0; k < BK / 16; k++)
                    umma(tmem_base, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), idesc, (kt > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty_bar[s]);
            }
            if (ok) umma_commit(&accum_bar);
        }
    } else {
        const int quad = warp & 3;
        const int n = n0 + quad * 32 + lane;  // this thread's weight row
        if (fold.stats_in != nullptr) {
            // The norm factors of the rows this CTA finishes: with several slices of K every splits-th one.  Warp q of the
            // four takes rows q, q + 4, ... of them, eight at a time so that their loads are in flight together; its lanes
            // add every 32nd partial sum of a row and a tree adds the lanes: an order that does not depend on the other rows.
            for (int k0 = quad; split + splits * k0 < M; k0 += 32) {
                float t[8];
#pragma unroll
                for (int u = 0; u < 8; u++) t[u] = 0.f;
#pragma unroll 2
                for (int c = lane; c < fold.stats_count; c += 32) {
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int b = split + splits * (k0 + 4 * u);
                        if (b < M) t[u] += fold.stats_in[(int64_t)b * fold.stats_in_stride + c];
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int b = split + splits * (k0 + 4 * u);
                    const float total = warp_sum(t[u]);
                    if (lane == 0 && b < M) rs_s[b] = 1.0f / sqrtf(total / (float)fold.norm_n + fold.eps);
                }
            }
            asm volatile("bar.sync 1, 128;\n" ::: "memory");  // the four epilogue warps
        }
        bool have = KT > 0;
        if (have && !mbar_wait(&accum_bar, 0)) {
            atomicCAS(&g_status, 0, 3);
            have = false;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (splits > 1) {
            // partial tile in this CTA's shared memory: part[b][row of the tile]; the operand
            // stages are free, every product that read them has completed
            constexpr int CH = NB < 32 ? 16 : 32;
            float* part = reinterpret_cast<float*>(tiles) + quad * 32 + lane;
#pragma unroll 1
            for (int c0 = 0; c0 < M; c0 += CH) {
                uint32_t r[CH];
                if (have) {
                    tmem_ld(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, r);
                } else {
#pragma unroll
                    for (int i = 0; i < CH; i++) r[i] = 0u;
                }
#pragma unroll
                for (int i = 0; i < CH; i++) part[(c0 + i) * BMW] = __uint_as_float(r[i]);
            }
        }
#pragma unroll 1
        for (int c0 = 0; c0 < NB; c0 += 16) {
            if (c0 >= M || splits > 1) break;
            uint32_t r[16];
            if (have) {
                tmem_ld16(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, r);
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) r[i] = 0u;
            }
            if (epi == 2) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int b = c0 + i;
                    float sq = 0.f;
                    if (b < M && n < N) {
                        float* hq = reinterpret_cast<float*>(Y) + (int64_t)b * ldy + n;
                        const float hn = *hq + __uint_as_float(r[i]);
                        *hq = hn;
                        sq = hn * hn;
                        if (fold.next_w != nullptr) fold.xn_out[(int64_t)b * fold.ldxn + n] = __float2bfloat16_rn(hn * fold.next_w[n]);
                    }
                    sq = warp_sum(sq);
                    if (lane == 0 && b < M) sq_part[quad][b] = sq;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float v = __uint_as_float(r[i]);
                    if (fold.stats_in != nullptr && c0 + i < M) v *= rs_s[c0 + i];
                    float other = __shfl_down_sync(0xffffffffu, v, 8);
                    if (c0 + i < M) store_out<TC>(Y, ldy, c0 + i, n, N, v, other, epi);
                }
            }
        }
        if (splits == 1 && epi == 2) {
            // the four warps' sums of each batch row, added in warp order
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
            const int b = (int)threadIdx.x - 64;
            if (b < M) fold.stats_out[(int64_t)b * fold.stats_out_stride + blockIdx.x] = (sq_part[0][b] + sq_part[1][b]) + (sq_part[2][b] + sq_part[3][b]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    if (splits == 1) {
        __syncthreads();
        if (warp == 1) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
        }
        return;
    }

    // All slices of the tile have left their partial tiles: add them.  CTA r of the cluster takes batch rows r, r + slices, ...: a
    // warp a row, a lane four neighbouring rows of the tile.  What the residual variant reads from global memory is requested
    // while the cluster gathers.  All slices of a row are asked for before the first is added, and added as they are: kept in the
    // warp's own shared memory first, for several rows at once, the products took up to a tenth longer (us a call in a chain, that
    // way and so: 9 x 1024 x 2048 4.6 and 4.2, 64 x 2048 x 6144 11.1 and 10.9, 256 x 2048 x 2048 14.6 and 11.8; a layer's four
    // products at 1.7B sizes, 16 rows 34.7 and 33.2, 32 39.6 and 38.9, 64 47.0 and 44.3).
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
    const int n = n0 + lane * 4, have = N - n;
    const int row_step = splits * (THREADS / 32);
    const int row0 = (int)rank + splits * warp;
    float4 ahead = make_float4(0.f, 0.f, 0.f, 0.f), next_w = ahead;   // epi 2: what the residual holds for the next row; the next norm's weight
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    if (epi == 2) {
        if (fold.next_w != nullptr) next_w = load4(fold.next_w + n, have, vec);
        if (row0 < M) ahead = load4(reinterpret_cast<const float*>(Y) + (int64_t)row0 * ldy + n, have, vec);
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (warp == 1) {
        // the barrier was also this CTA's: its epilogue warps have read the accumulators
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    const uint32_t part_addr = s32(tiles) + (uint32_t)(lane * 16);
#pragma unroll 1
    for (int bb = row0; bb < M; bb += row_step) {
        float4 x[MAX_SPLITS];
#pragma unroll
        for (int sl = 0; sl < MAX_SPLITS; sl++) {
            if (sl >= splits) break;
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(part_addr + (uint32_t)(bb * BMW * 4)), "r"(sl));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(x[sl].x), "=f"(x[sl].y), "=f"(x[sl].z), "=f"(x[sl].w) : "r"(remote) : "memory");
        }
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int sl = 0; sl < MAX_SPLITS; sl++) {
            if (sl >= splits) break;
            v.x += x[sl].x;
            v.y += x[sl].y;
            v.z += x[sl].z;
            v.w += x[sl].w;
        }
        if (bb + row_step >= M) {
            // this warp reads no other CTA's memory any more
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        }
        if (epi == 2) {
            float* hq = reinterpret_cast<float*>(Y) + (int64_t)bb * ldy + n;
            const float4 h = make_float4(ahead.x + v.x, ahead.y + v.y, ahead.z + v.z, ahead.w + v.w);
            if (bb + row_step < M) ahead = load4(hq + (int64_t)row_step * ldy, have, vec);
            store4(hq, h, have, vec);
            if (fold.next_w != nullptr) store4(fold.xn_out + (int64_t)bb * fold.ldxn + n, make_float4(h.x * next_w.x, h.y * next_w.y, h.z * next_w.z, h.w * next_w.w), have, vec);
            // columns behind the last are zero.  The lanes of the warp hold the whole tile's share of this batch row
            float sq = h.x * h.x;
            sq += h.y * h.y;
            sq += h.z * h.z;
            sq += h.w * h.w;
            sq = warp_sum(sq);
            if (lane == 0) fold.stats_out[(int64_t)bb * fold.stats_out_stride + blockIdx.x] = sq;
            continue;
        }
        if (fold.stats_in != nullptr) {
            const float rs = rs_s[bb];
            v = make_float4(v.x * rs, v.y * rs, v.z * rs, v.w * rs);
        }
        if (epi == 0) {
            store4(Y + (int64_t)bb * ldy + n, v, have, vec);
        } else {
            // The up rows of four gate rows are eight rows on: two lanes on.  Each of the two lanes finishes two of the four.
            const bool is_up = lane & 2;
            const float give0 = is_up ? v.x : v.z, give1 = is_up ? v.y : v.w;
            const float got0 = __shfl_xor_sync(0xffffffffu, give0, 2), got1 = __shfl_xor_sync(0xffffffffu, give1, 2);
            const float z0 = silu_f(is_up ? got0 : v.x) * (is_up ? v.z : got0), z1 = silu_f(is_up ? got1 : v.y) * (is_up ? v.w : got1);
            const int col = ((n >> 4) << 3) + (n & 7) + (is_up ? 2 : 0);
            if (n < N) store2(Y + (int64_t)bb * ldy + col, z0, z1, vec);   // N is a multiple of 16
        }
    }
    // no CTA may leave while another still reads its shared memory
    __syncwarp();
    if (row0 >= M) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

constexpr int MAX_TILES = 8192;
constexpr int UNEVEN_TILES = 148;  // more tiles than this many SMs: see dispatch()

template <typename TC, int NB, int STAGES>
int launch(const void* X, const void* W, void* Y, int M, int N, int K, int64_t ldx, int64_t ldy, int epi, int splits,
           const DecodeFold& fold, cudaStream_t stream) {
    constexpr int X_BYTES = NB * BK * 2;
    int smem = STAGES * (W_BYTES + X_BYTES) + 1024;
    const int part = NB * BMW * 4 + 1024;
    if (part > smem) smem = part;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc5_decode_kernel<TC, NB, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) GB_REFUSE("gemm_tc5_decode: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    CUtensorMap map_w, map_x;
    if (int rc = tc5_make_map(&map_w, W, N, K, K, BMW)) return rc;
    if (int rc = tc5_make_map(&map_x, X, M, K, ldx, NB)) return rc;
    const int tiles = ceil_div(N, BMW);
    const int KB = ceil_div(K, BK);
    while (splits > 1 && KB < splits) splits >>= 1;
    const int kb_per_split = ceil_div(KB, splits);
    const uintptr_t rows = (uintptr_t)Y | (uintptr_t)fold.next_w | (uintptr_t)fold.xn_out | ((uintptr_t)(ldy | fold.ldxn) * 4);
    const int vec = !(rows & 15);   // four neighbouring elements of every row in one access
    if (tiles > MAX_TILES) GB_REFUSE("gemm_tc5_decode: N = %d exceeds %d tiles", N, MAX_TILES);
    cudaError_t e = launch_pdl_cluster(gemm_tc5_decode_kernel<TC, NB, STAGES>, dim3(tiles, splits), dim3(THREADS), (size_t)smem, stream, 1,
                                       (unsigned)splits, map_w, map_x, (TC*)Y, M, N, K, ldy, splits, kb_per_split, epi, vec, fold);
    if (e != cudaSuccess) GB_REFUSE("gemm_tc5_decode: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

template <typename TC>
int dispatch(const void* X, const void* W, void* Y, int M, int N, int K, int64_t ldx, int64_t ldy, int epi, int splits,
             const DecodeFold& fold, cudaStream_t stream) {
    if (M <= 16) return launch<TC, 16, 4>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
    // More tiles than SMs but fewer than two to an SM (the gate/up product of an 8B layer: 192 tiles on
    // 148 SMs): some SMs would stream two tiles while most stream one.  Such a product runs in two K
    // slices with three stages, so that three CTAs fit an SM and every SM gets two or three of the
    // smaller pieces (64 rows: 50.7 -> 43.3 us; 33 rows: 43.5 -> 38.4 us).
    const bool uneven = splits == 2 && ceil_div(N, BMW) > UNEVEN_TILES;
    if (M <= 32) {
        if (uneven) return launch<TC, 32, 3>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
        return launch<TC, 32, 4>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
    }
    if (M <= 64) {
        if (uneven) return launch<TC, 64, 3>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
        return launch<TC, 64, 4>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
    }
    if (M <= 128) return launch<TC, 128, 3>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
    return launch<TC, 256, 3>(X, W, Y, M, N, K, ldx, ldy, epi, splits, fold, stream);
}

}  // namespace

// How many slices of K (1, 2, 4 or 8, the size of the cluster) the kernel would like for M rows of
// this shape on a device with `sms` SMs, two CTAs to an SM.
//   More than 16 rows: the most slices that keep at most about 2 * sms CTAs and at least eight K
//   steps of 64 a slice; CTAs that queue behind a full machine cost more than they gain (24576 x 4096
//   at 64 rows: 40.8 us whole, 57.6 us in two slices).
//   Up to 16 rows a CTA is lighter and a short queue pays: a CTA's time is its K steps plus about
//   eight steps of fixed cost, and the choice minimises queue depth x CTA time (24576 x 4096 at 16
//   rows: 36.5 us in two slices, 38.0 whole, 39.3 in four).
GB_API int gb_gemm_tc5_decode_splits(int M, int N, int K, int sms) {
    const int tiles = ceil_div(N, BMW), KB = ceil_div(K, BK);
    if (sms <= 0) sms = 1;
    if (M > 16) {
        int per_sm = M > 128 ? 1 : 2;  // CTAs that fit on an SM with the operand stages of this many rows
        if (M <= 64 && tiles > UNEVEN_TILES && tiles > sms && tiles < 2 * sms) per_sm = 3;  // see dispatch(): three stages
        int want = (per_sm * sms) / (tiles > 0 ? tiles : 1);
        if (want > KB / 8) want = KB / 8;
        int s = 1;
        while (s * 2 <= want && s < 8) s *= 2;
        return s;
    }
    int best = 1;
    double best_cost = 0.0;
    for (int s = 1; s <= 8; s *= 2) {
        if (s > 1 && KB / s < 1) break;
        const double queue = tiles * (double)s / (2.0 * sms);
        const double cost = (queue > 1.0 ? queue : 1.0) * ((double)ceil_div(KB, s) + 8.0);
        if (s == 1 || cost < best_cost) {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

static int decode_checks(const char* who, const void* X, const void* W, int M, int N, int K, int64_t ldx, int splits) {
    if (M > 256) GB_REFUSE("%s: %d rows; this kernel takes at most 256", who, M);
    if (K <= 0 || (K & 7)) GB_REFUSE("%s: K = %d must be a positive multiple of 8", who, K);
    if ((ldx & 7) || ldx < K) GB_REFUSE("%s: row stride %lld of X must be a multiple of 8 and at least K", who, (long long)ldx);
    if (((uintptr_t)X & 15) || ((uintptr_t)W & 15)) GB_REFUSE("%s: operands must be 16-byte aligned", who);
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8) GB_REFUSE("%s: %d slices; 1, 2, 4 or 8", who, splits);
    return 0;
}

// epi = 0: Y[M, N].  epi = 1: Y[M, N / 2] = silu(gate) * up with gate/up rows of W interleaved in
// blocks of eight.  splits: 1, 2, 4 or 8 slices of K (the size of the cluster).
GB_API int gb_gemm_tc5_decode(const void* X, const void* W, void* Y, int c_dtype, int M, int N, int K, int64_t ldx, int64_t ldy,
                              int epi, int splits, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const char* who = "gemm_tc5_decode";
    if (int rc = decode_checks(who, X, W, M, N, K, ldx, splits)) return rc;
    if (epi == 0 && ldy < N) GB_REFUSE("%s: row stride %lld of Y is shorter than N = %d", who, (long long)ldy, N);
    if (epi == 1 && ((N & 15) || ldy < N / 2)) GB_REFUSE("%s: the SwiGLU epilogue needs N = %d to be a multiple of 16", who, N);
    if (epi != 0 && epi != 1) GB_REFUSE("%s: unknown epilogue %d", who, epi);
    const DecodeFold none = {};
    if (c_dtype == GB_F32) return dispatch<float>(X, W, Y, M, N, K, ldx, ldy, epi, splits, none, stream);
    if (c_dtype == GB_BF16) return dispatch<__nv_bfloat16>(X, W, Y, M, N, K, ldx, ldy, epi, splits, none, stream);
    GB_REFUSE("%s: unknown output dtype %d", who, c_dtype);
}

// The consumer of prescaled rows (see gemm_skinny_fold.cu) for 9 to 64 rows: Y = rs[row] * (X W^T),
// plain (swiglu 0) or through the SwiGLU epilogue, rs from stats_in[row][0 .. stats_count).
GB_API int gb_gemm_tc5_decode_scaled(const void* X, int64_t ldx, float eps, const float* stats_in, int stats_count,
                                     int64_t stats_in_stride, const void* W, void* Y, int c_dtype, int64_t ldy, int M, int N, int K,
                                     int swiglu, int splits, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const char* who = "gemm_tc5_decode_scaled";
    if (int rc = decode_checks(who, X, W, M, N, K, ldx, splits)) return rc;
    if (M > FOLD_ROWS) GB_REFUSE("%s: %d rows; the folded variants take at most %d", who, M, FOLD_ROWS);
    if (!stats_in || stats_count <= 0 || stats_in_stride < stats_count) GB_REFUSE("%s: %d partial sums a row with a row stride of %lld", who, stats_count, (long long)stats_in_stride);
    if (!swiglu && ldy < N) GB_REFUSE("%s: row stride %lld of Y is shorter than N = %d", who, (long long)ldy, N);
    if (swiglu && ((N & 15) || ldy < N / 2)) GB_REFUSE("%s: the SwiGLU epilogue needs N = %d to be a multiple of 16", who, N);
    DecodeFold fold = {};
    fold.stats_in = stats_in;
    fold.stats_count = stats_count;
    fold.stats_in_stride = stats_in_stride;
    fold.eps = eps;
    fold.norm_n = K;
    if (c_dtype == GB_F32) return dispatch<float>(X, W, Y, M, N, K, ldx, ldy, swiglu ? 1 : 0, splits, fold, stream);
    if (c_dtype == GB_BF16) return dispatch<__nv_bfloat16>(X, W, Y, M, N, K, ldx, ldy, swiglu ? 1 : 0, splits, fold, stream);
    GB_REFUSE("%s: unknown output dtype %d", who, c_dtype);
}

// The producer for 9 to 64 rows: Hres[M, N] += X W^T (fp32 residual, in place); stats_out[row][c] =
// the sum of squares of the new values of the row in columns 128 c .. 128 c + 127; and, if next_w is
// given, xn_out = bf16(Hres * next_w).  *stats_count receives the number of such tiles.
GB_API int gb_gemm_tc5_decode_residual(const void* X, int64_t ldx, const void* W, float* Hres, int64_t ldh, float* stats_out,
                                       int64_t stats_out_stride, int* stats_count, const float* next_w, void* xn_out, int64_t ldxn,
                                       int M, int N, int K, int splits, cudaStream_t stream) {
    const int count = ceil_div(N, BMW);
    if (stats_count) *stats_count = count;
    if (M <= 0 || N <= 0) return 0;
    const char* who = "gemm_tc5_decode_residual";
    if (int rc = decode_checks(who, X, W, M, N, K, ldx, splits)) return rc;
    if (M > FOLD_ROWS) GB_REFUSE("%s: %d rows; the folded variants take at most %d", who, M, FOLD_ROWS);
    if (ldh < N) GB_REFUSE("%s: row stride %lld of the residual is shorter than N = %d", who, (long long)ldh, N);
    if (!stats_out || stats_out_stride < count) GB_REFUSE("%s: the statistics buffer needs %d floats a row", who, count);
    if (next_w && (!xn_out || ldxn < N)) GB_REFUSE("%s: the next norm's weight is given without room for its %d-wide rows", who, N);
    DecodeFold fold = {};
    fold.stats_out = stats_out;
    fold.stats_out_stride = stats_out_stride;
    fold.next_w = next_w;
    fold.xn_out = (__nv_bfloat16*)xn_out;
    fold.ldxn = ldxn;
    return dispatch<float>(X, W, Hres, M, N, K, ldx, ldh, 2, splits, fold, stream);
}

GB_API int gb_gemm_tc5_decode_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_status, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_status, &zero, sizeof(int));
    return v;
}
