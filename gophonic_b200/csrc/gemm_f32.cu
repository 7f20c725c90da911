// C[M, N] = A[M, K] * W[N, K]^T, all float32, on the CUDA cores: the products of the true 32-bit path.
//
// Every output element is the sum over k in ascending order in one fp32 accumulator, as in
// gemm_simt.cu, whatever M is and whichever kernel or tile takes it: rows do not depend on what else
// is in the batch.  That order rules out cutting K, so both kernels spread outputs, not K.
//
// Few rows (single tokens, short prompts): bound by reading W once, and by a lane's chain of additions, 4
// cycles a column of K.  A CTA owns nt columns of the output, nt chosen so that the CTAs fill the SMs in
// whole waves, and streams its nt weight rows and the activations through shared memory in stages of KS
// columns, several stages in flight; a thread owns one column and MPT rows.  An ordinary launch: W may be what the
// kernel ahead makes, and as a dependent launch the waiting CTAs took the place of those at work (three rows behind a
// norm, 12288 x 2048: 41.0 us, with the weights requested ahead of the wait or not, and 30.8 so).  Three rows, one product behind
// the other inside a graph, against tiles of 64 x 64 without any stages ahead (us; floor of the weights' bytes): 4096 x 2048 160
// -> 13.5 (5), 12288 x 2048 219 -> 28 (15), 2048 x 6144 473 -> 27 (8), 151936 x 2048 1407 -> 220 (190).
//
// More rows: bound by the multiply-add rate.  Tiles of BM x BN in registers, operands transposed on their way
// into shared memory, the global loads two stages and the fragments one column ahead of their use, two
// columns of the output per fma.rn.f32x2 (with scalar multiply-adds the same tile took 1 to 10 % longer).  341
// rows: 12288 x 2048 784 -> 367 us, 2048 x 6144 614 -> 334; 1024 rows, 12288 x 2048: 2022 -> 1001 us, 51
// TFLOP/s.  What is left there is latency (a stage of a lone 64 x 64 tile takes 0.6 us, its arithmetic 0.27)
// and the last wave: a single accumulator in order of k leaves no K to cut.
#include "mma.cuh"
#include "api.h"

namespace {

// ---- few rows -----------------------------------------------------------------------------
constexpr int ROWS_THREADS = 256;
constexpr int ROWS_MAX = 64;
constexpr int ROWS_COLS = 96;           // columns a CTA at most
constexpr int ROWS_SMEM = 104 * 1024;  // of two CTAs an SM

template <int MPT, int KS>
__global__ void __launch_bounds__(ROWS_THREADS) gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                     float* __restrict__ C, int M, int N, int K, int64_t lda,
                                                                     int64_t ldw, int64_t ldc, int nt, int stages) {
    extern __shared__ float sm[];
    constexpr int PITCH = KS + 4;   // 16-byte chunks a row: odd, so that eight lanes on eight rows meet no bank twice
    constexpr int CH = KS / 4;
    const int stage_floats = (nt + M) * PITCH;
    const int n0 = blockIdx.x * nt;
    const int tid = threadIdx.x;
    const int steps = (K + KS - 1) / KS;

    // where the arithmetic fits four warps, the other four do the fetching
    const int groups = (M + MPT - 1) / MPT;
    const int first_loader = nt * groups <= ROWS_THREADS / 2 ? ROWS_THREADS / 2 : 0, loaders = ROWS_THREADS - first_loader;
    auto load = [&](const float* src, int64_t ld, int rows, int rows_all, int first, float* dst, int s) {
        if (tid < first_loader) return;
        for (int c = tid - first_loader; c < rows * CH; c += loaders) {
            const int r = c / CH, q = c % CH, k = s * KS + q * 4;
            const int row = first + r < rows_all ? first + r : rows_all - 1;
            const bool in = k < K;  // K is a multiple of 4: a chunk is wholly inside or wholly outside
            cp_async16(dst + r * PITCH + q * 4, src + (int64_t)row * ld + (in ? k : 0), in ? 16 : 0);
        }
    };
    const int ahead = stages - 1;
    for (int s = 0; s < ahead; s++) {
        if (s < steps) {
            load(W, ldw, nt, N, n0, sm + s * stage_floats, s);
            load(A, lda, M, M, 0, sm + s * stage_floats + nt * PITCH, s);
        }
        cp_async_commit();
    }

    const bool works = tid < nt * groups;
    const int n = tid % nt, mg = works ? tid / nt : 0;
    float acc[MPT];
    int xo[MPT];
#pragma unroll
    for (int i = 0; i < MPT; i++) {
        acc[i] = 0.f;
        const int m = mg * MPT + i;
        xo[i] = (nt + (m < M ? m : M - 1)) * PITCH;
    }
    for (int s = 0; s < steps; s++) {
        // one group was committed per stage, empty ones behind the last: stage s has landed when at most
        // ahead - 1 are open
        switch (ahead) {
            case 1: cp_async_wait<0>(); break;
            case 2: cp_async_wait<1>(); break;
            case 3: cp_async_wait<2>(); break;
            case 4: cp_async_wait<3>(); break;
            case 5: cp_async_wait<4>(); break;
            case 6: cp_async_wait<5>(); break;
            default: cp_async_wait<6>(); break;
        }
        __syncthreads();  // stage s is visible to all, and all are done with stage s - 1
        if (s + ahead < steps) {
            float* dst = sm + ((s + ahead) % stages) * stage_floats;
            load(W, ldw, nt, N, n0, dst, s + ahead);
            load(A, lda, M, M, 0, dst + nt * PITCH, s + ahead);
        }
        cp_async_commit();
        if (works) {
            const float* base = sm + (s % stages) * stage_floats;
            const float* w = base + n * PITCH;
            // the next U chunks of four columns are read while these are multiplied
            constexpr int U = MPT <= 2 ? 4 : MPT == 4 ? 2 : 1, CHUNKS = KS / (4 * U);
            float4 wv[2][U], xv[2][MPT][U];
            auto read = [&](int buf, int c) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    wv[buf][u] = *(const float4*)(w + (c * U + u) * 4);
#pragma unroll
                    for (int i = 0; i < MPT; i++) xv[buf][i][u] = *(const float4*)(base + xo[i] + (c * U + u) * 4);
                }
            };
            read(0, 0);
#pragma unroll
            for (int c = 0; c < CHUNKS; c++) {
                if (c + 1 < CHUNKS) read((c + 1) & 1, c + 1);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const float4 a = wv[c & 1][u];
#pragma unroll
                    for (int i = 0; i < MPT; i++) acc[i] = fmaf(xv[c & 1][i][u].x, a.x, acc[i]);
#pragma unroll
                    for (int i = 0; i < MPT; i++) acc[i] = fmaf(xv[c & 1][i][u].y, a.y, acc[i]);
#pragma unroll
                    for (int i = 0; i < MPT; i++) acc[i] = fmaf(xv[c & 1][i][u].z, a.z, acc[i]);
#pragma unroll
                    for (int i = 0; i < MPT; i++) acc[i] = fmaf(xv[c & 1][i][u].w, a.w, acc[i]);
                }
            }
        }
    }
    if (works && n0 + n < N) {
#pragma unroll
        for (int i = 0; i < MPT; i++) {
            const int m = mg * MPT + i;
            if (m < M) C[(int64_t)m * ldc + n0 + n] = acc[i];
        }
    }
}

template <int MPT, int KS>
int launch_rows_ks(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, int nt,
                   cudaStream_t stream) {
    const int stage = (nt + M) * (KS + 4) * 4;
    int stages = ROWS_SMEM / stage;
    stages = stages > 8 ? 8 : stages;   // never below 2: see launch_rows
    static bool configured[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) GB_REFUSE("gemm_f32: no current device");
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MPT, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM);
        if (e != cudaSuccess) GB_REFUSE("gemm_f32: cannot reserve %d bytes of shared memory: %s", ROWS_SMEM, cudaGetErrorString(e));
        configured[dev] = true;
    }
    gemm_f32_rows_kernel<MPT, KS><<<ceil_div(N, nt), ROWS_THREADS, (size_t)stages * stage, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, nt, stages);
    GB_CHECK_LAUNCH("gemm_f32");
    return 0;
}

template <int MPT>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, cudaStream_t stream) {
    // columns a CTA: as many as its threads and shared memory hold, evened out over whole waves of the SMs
    const int sms = gb_sm_count(), groups = ceil_div(M, MPT);
    int most = ROWS_THREADS / groups;
    if (most > ROWS_COLS) most = ROWS_COLS;
    const int waves = ceil_div(N, sms * most);
    const int nt = ceil_div(N, sms * waves);
    // nt + M is at most 96 + 64: two stages of 64 columns take at most 85 KB
    if (nt + M <= 24) return launch_rows_ks<MPT, 256>(A, W, C, M, N, K, lda, ldw, ldc, nt, stream);
    if (nt + M <= 48) return launch_rows_ks<MPT, 128>(A, W, C, M, N, K, lda, ldw, ldc, nt, stream);
    return launch_rows_ks<MPT, 64>(A, W, C, M, N, K, lda, ldw, ldc, nt, stream);
}

// ---- tiles --------------------------------------------------------------------------------
constexpr int BK = 16;

__device__ __forceinline__ unsigned long long dup2(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// A warp's lanes stand 4 x 8; a lane owns TM / 4 groups of four rows, 16 apart, and TN / 4 groups of four
// columns, 32 apart.
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), (TN == 8 ? 384 : 512) / ((BM / TM) * (BN / TN)))
    gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int64_t lda,
                         int64_t ldw, int64_t ldc, int vec_out) {
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int WN = BN / (8 * TN);                 // warps along the columns
    constexpr int LA = BM * 4 / THREADS, LW = BN * 4 / THREADS;
    static_assert(BM * 4 % THREADS == 0 && BN * 4 % THREADS == 0, "whole rounds of loads");
    __shared__ float As[2][BK][BM];
    __shared__ float Ws[2][BK][BN];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int wm = (warp / WN) * 4 * TM, wn = (warp % WN) * 8 * TN;
    const int am = wm + (lane >> 3) * 4, wc = wn + (lane & 7) * 4;

    // thread -> (row, four columns of K): four lanes read 64 contiguous bytes of a row.  A value goes to
    // [k][row ^ 8 (k / 4)]: the four lanes of a row and the eight rows of a warp meet no bank twice.
    const int q = tid & 3, r0 = tid >> 2;
    float4 ra2[2][LA], rw2[2][LW];
    auto fetch = [&](int k0, int h) {
        float4 (&ra)[LA] = ra2[h];
        float4 (&rw)[LW] = rw2[h];
        const int k = k0 + q * 4;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int m = m0 + r0 + i * (THREADS / 4);
            ra[i] = m < M && k < K ? *(const float4*)(A + (int64_t)m * lda + k) : z;
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int n = n0 + r0 + i * (THREADS / 4);
            rw[i] = n < N && k < K ? __ldg((const float4*)(W + (int64_t)n * ldw + k)) : z;
        }
    };
    auto place = [&](int b, int h) {
        float4 (&ra)[LA] = ra2[h];
        float4 (&rw)[LW] = rw2[h];
#pragma unroll
        for (int i = 0; i < LA; i++) {
            const int r = (r0 + i * (THREADS / 4)) ^ (8 * q);
            As[b][q * 4 + 0][r] = ra[i].x;
            As[b][q * 4 + 1][r] = ra[i].y;
            As[b][q * 4 + 2][r] = ra[i].z;
            As[b][q * 4 + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LW; i++) {
            const int r = (r0 + i * (THREADS / 4)) ^ (8 * q);
            Ws[b][q * 4 + 0][r] = rw[i].x;
            Ws[b][q * 4 + 1][r] = rw[i].y;
            Ws[b][q * 4 + 2][r] = rw[i].z;
            Ws[b][q * 4 + 3][r] = rw[i].w;
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++) {
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;
    }

    float a[2][TM];
    unsigned long long w[2][TN / 2];
    auto read = [&](int buf, int b, int kk) {
#pragma unroll
        for (int i = 0; i < TM / 4; i++) *(float4*)(a[buf] + 4 * i) = *(const float4*)&As[b][kk][(am + 16 * i) ^ (8 * (kk / 4))];
#pragma unroll
        for (int j = 0; j < TN / 4; j++) *(ulonglong2*)(w[buf] + 2 * j) = *(const ulonglong2*)&Ws[b][kk][(wc + 32 * j) ^ (8 * (kk / 4))];
    };
    auto compute = [&](int b) {
        read(0, b, 0);
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            if (kk + 1 < BK) read((kk + 1) & 1, b, kk + 1);
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const unsigned long long aa = dup2(a[kk & 1][i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) fma2(acc[i][j], aa, w[kk & 1][j]);
            }
        }
    };

    fetch(0, 0);
    place(0, 0);
    fetch(BK, 0);
    __syncthreads();
    // the loads of the stage after next are issued before this one is multiplied
    for (int k0 = 0; k0 < K; k0 += 2 * BK) {
        fetch(k0 + 2 * BK, 1);
        compute(0);
        place(1, 0);
        __syncthreads();
        if (k0 + BK >= K) break;
        fetch(k0 + 3 * BK, 0);
        compute(1);
        place(0, 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + am + 16 * (i / 4) + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 4; j++) {
            const int n = n0 + wc + 32 * j;
            float* c = C + (int64_t)m * ldc + n;
            float4 v;
            *(unsigned long long*)&v.x = acc[i][2 * j];
            *(unsigned long long*)&v.z = acc[i][2 * j + 1];
            if (vec_out && n + 3 < N) {
                *(float4*)c = v;
            } else {
                if (n < N) c[0] = v.x;
                if (n + 1 < N) c[1] = v.y;
                if (n + 2 < N) c[2] = v.z;
                if (n + 3 < N) c[3] = v.w;
            }
        }
    }
}

template <int BM, int BN, int TM, int TN>
int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, cudaStream_t stream) {
    const dim3 grid(ceil_div(M, BM), ceil_div(N, BN));  // tiles of the same weight rows beside each other: W comes from HBM once
    if (grid.y > 65535) GB_REFUSE("gemm_f32: %d columns exceed one launch", N);
    const int vec_out = (ldc & 3) == 0 && !((uintptr_t)C & 15);
    gemm_f32_tile_kernel<BM, BN, TM, TN><<<grid, (BM / TM) * (BN / TN), 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, vec_out);
    GB_CHECK_LAUNCH("gemm_f32");
    return 0;
}

}  // namespace

// Rows of 16-byte chunks, and few enough columns for one launch of the narrowest tile.
bool gb_gemm_f32_accepts(const void* A, const void* W, int N, int K, int64_t lda, int64_t ldw) {
    return (K & 3) == 0 && (lda & 3) == 0 && (ldw & 3) == 0 && !((uintptr_t)A & 15) && !((uintptr_t)W & 15) && N <= 65535 * 64;
}

int gb_gemm_f32_launch(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, cudaStream_t stream) {
    const int sms = gb_sm_count();
    // Few rows: as few rows a thread as leave the arithmetic on four warps, one a scheduler (three rows of
    // 4096 columns: 20.5 us with one row a thread, 22.5 with two, 28.7 with four; of 12288: 38.9, 45.1, 36.9).
    // Where even eight rows a thread do not, the kernel is ahead of the tiles up to 16 rows only (12288 columns,
    // 16 rows: 71 against 81 us; 24 rows: 82 against 82).
    if (M <= ROWS_MAX) {
        const int nt = ceil_div(N, sms * ceil_div(N, sms * ROWS_COLS));
        if (nt * M <= 128) return launch_rows<1>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (nt * ceil_div(M, 2) <= 128) return launch_rows<2>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (nt * ceil_div(M, 4) <= 128) return launch_rows<4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (nt * ceil_div(M, 8) <= 128) return launch_rows<8>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (M <= 16) return launch_rows<4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
    // The tile: what the busiest SM's tiles take, from one alone and from several side by side (us at K = 2048).
    struct Tile {
        int bm, bn, alone, each;
    };
    static const Tile tiles[4] = {{128, 128, 184, 184}, {64, 128, 115, 97}, {64, 64, 78, 56}, {32, 64, 63, 41}};
    int64_t best = INT64_MAX;
    int pick = 0;
    for (int i = 0; i < 4; i++) {
        const int64_t n = ((int64_t)ceil_div(M, tiles[i].bm) * ceil_div(N, tiles[i].bn) + sms - 1) / sms;
        const int64_t t = n * tiles[i].each > tiles[i].alone ? n * tiles[i].each : tiles[i].alone;
        if (t < best) {
            best = t;
            pick = i;
        }
    }
    switch (pick) {
        case 0: return launch_tile<128, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        case 1: return launch_tile<64, 128, 8, 8>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        case 2: return launch_tile<64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        default: return launch_tile<32, 64, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
}
