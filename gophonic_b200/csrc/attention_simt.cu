// Causal grouped-query attention over the paged cache on the CUDA cores, all arithmetic fp32.
//
// It is the attention of the true 32-bit path for prompts and for single tokens, and the
// fallback of the bfloat16 path for head sizes the tensor-core kernels do not take.  A CTA owns
// one (sequence, kv head, tile of query rows); its 16 rows are (query position, head of the
// group) pairs, so the heads of a group share every key/value tile that is read
// (internal/qwen3lm/gpu.metal:1102-1234 shares tiles the same way).  Keys are visited in tiles of
// 32 that start at absolute positions 0, 32, 64, ..., with a streaming softmax
// (internal/qwen3lm/ops.go:259-293): a row's result does not depend on how its sequence was cut
// into steps or on what else is in the batch.
#include "mma.cuh"
#include "api.h"

#include <math.h>

#include <type_traits>


namespace {

constexpr int RW = 4;       // rows per warp
constexpr int ROWS = 16;    // rows per CTA (4 warps)
constexpr int KT = 32;      // keys per tile
constexpr int SIMT_MAX_D = 640;    // widest key head (a latent of 512 and 128 rotated channels); what one CTA stages
constexpr int SIMT_MAX_DV = 512;   // widest value head

// What both kernels of this file share, so that a row's keys, their order and its sums are the same in either.

// The tiles of keys that a CTA's rows q0 .. last_q visit in its share of the splits.  With kept first tokens they are those of
// keys [0, keep_first) and then those of the window, each once and in order of position: tile index i < n_first is tile i, the
// others follow from t_lo.
struct KeyTiles {
    int t_lo, n_first, my_lo, my_hi;
    __device__ __forceinline__ KeyTiles(const AttnParamsX& p, int past, int q0, int last_q, int split) {
        int lo_pos = 0;
        if (p.window > 0) {
            lo_pos = past + q0 - p.window + 1;
            if (lo_pos < 0) lo_pos = 0;
        }
        if (p.chunk > 0) {
            // the block of the tile's first row begins no later than any other row's
            const int b = (past + q0) - (past + q0) % p.chunk;
            if (b > lo_pos) lo_pos = b;
        }
        t_lo = lo_pos / KT;
        n_first = p.window > 0 && p.keep_first > 0 ? (p.keep_first + KT - 1) / KT : 0;
        if (n_first > t_lo) n_first = t_lo;
        const int n_tiles = n_first + ((past + last_q) / KT + 1 - t_lo);
        const int per = (n_tiles + p.num_splits - 1) / p.num_splits;
        my_lo = split * per;
        my_hi = my_lo + per < n_tiles ? my_lo + per : n_tiles;
    }
    __device__ __forceinline__ int tile(int i) const { return i < n_first ? i : t_lo + (i - n_first); }
};

__device__ __forceinline__ bool sees(const AttnParamsX& p, int pos, int key) {
    return key <= pos && (p.window <= 0 || key > pos - p.window || key < p.keep_first) && (p.chunk <= 0 || key >= pos - pos % p.chunk);
}

// One tile's scores of a row, a key a lane, into its running maximum and sum; the lane's weight.
template <int NE>
__device__ __forceinline__ float weigh(bool valid, float score, float& m, float& l, float (&acc)[NE]) {
    const float sv = valid ? score : -INFINITY;
    const float m_new = fmaxf(m, warp_max(sv));
    if (m_new == -INFINITY) return 0.f;
    const float corr = expf(m - m_new);
    const float pv = valid ? expf(sv - m_new) : 0.f;
    l = l * corr + warp_sum(pv);
#pragma unroll
    for (int e = 0; e < NE; e++) acc[e] *= corr;
    m = m_new;
    return pv;
}

// A finished row: divided by its sum, or as it is into the scratch memory of the splits.
template <typename T, int NE>
__device__ __forceinline__ void leave_row(const AttnParamsX& p, int seq, int split, int64_t row, int head, int dv, int lane, float m, float l,
                                          const float (&acc)[NE]) {
    if (p.num_splits == 1) {
        T* op = (T*)p.out + row * p.out_row_stride + (int64_t)head * dv;
        float lsum = l, keep = 1.f;
        if (p.sink) {
            // one more term in the denominator: a key that has no value, of score 0 or the head's own
            const float z = p.sinks ? p.sinks[head] : 0.f;
            const float mf = fmaxf(m, z);
            keep = expf(m - mf);
            lsum = lsum * keep + expf(z - mf);
        }
        const float inv = keep / lsum;
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int c = lane + 32 * e;
            if (c < dv) op[c] = from_f32<T>(acc[e] * inv);
        }
    } else {
        float* sp = p.scratch + (((int64_t)seq * p.heads + head) * p.num_splits + split) * (dv + 2);
        if (lane == 0) {
            sp[0] = m;
            sp[1] = l;
        }
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int c = lane + 32 * e;
            if (c < dv) sp[2 + c] = acc[e];
        }
    }
}

template <typename T, int NE>
__global__ void __launch_bounds__(128) attn_simt_kernel(AttnParamsX p) {
    extern __shared__ float sm[];
    const int d = p.d, ks = d + 1;
    const int dv = p.dv > 0 ? p.dv : p.d, vs = dv + 1;   // values may be narrower or wider than keys
    const int64_t v_tok = p.v_row_stride > 0 ? p.v_row_stride : dv;   // a value plane may be a view of wider rows
    float* Qs = sm;                // [16][d], pre-scaled
    float* Ks = Qs + ROWS * d;     // [32][d + 1]
    float* Vs = Ks + KT * ks;      // [32][dv + 1]

    const int G = p.heads / p.kv_heads;
    const int GC = G < ROWS ? G : ROWS;
    const int hchunks = (G + GC - 1) / GC;
    const int QT = ROWS / GC;

    const int seq = blockIdx.z / p.num_splits, split = blockIdx.z % p.num_splits;
    const int kvh = blockIdx.y / hchunks, chunk = blockIdx.y % hchunks;
    // consecutive key heads may read one value head: -1 if every key head has its own
    const int v_heads = p.v_share > 1 ? p.kv_heads / p.v_share : p.kv_heads, vh = p.v_share > 1 ? kvh / p.v_share : -1;
    const int q_len = p.seq_q_len[seq], kv_len = p.seq_kv_len[seq];
    const int q0 = blockIdx.x * QT;
    if (q0 >= q_len) return;
    const int past = kv_len - q_len;
    const int q_start = p.seq_q_start[seq];
    const int* bt = block_table_row(p.block_table, p.bt_stride, p.seq_slot[seq], p.max_slots);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // stage the query rows, scaled
    for (int idx = tid; idx < ROWS * d; idx += 128) {
        int r = idx / d, c = idx - r * d;
        int qi = r / GC, hg = chunk * GC + r % GC;
        bool ok = qi < QT && q0 + qi < q_len && hg < G;
        float v = 0.f;
        if (ok) {
            const T* qp = (const T*)p.q + (int64_t)(q_start + q0 + qi) * p.q_row_stride + (int64_t)(kvh * G + hg) * d;
            v = to_f32<T>(qp[c]) * p.scale;
        }
        Qs[idx] = v;
    }

    int row_pos[RW], row_head[RW], row_q[RW];
    bool row_ok[RW];
#pragma unroll
    for (int rr = 0; rr < RW; rr++) {
        int r = warp * RW + rr;
        int qi = r / GC, hg = chunk * GC + r % GC;
        row_ok[rr] = qi < QT && q0 + qi < q_len && hg < G;
        row_q[rr] = q0 + qi;
        row_head[rr] = kvh * G + hg;
        row_pos[rr] = past + q0 + qi;
    }

    const int last_q = (q0 + QT < q_len ? q0 + QT : q_len) - 1;
    const int hi_pos = past + last_q;
    const KeyTiles tiles(p, past, q0, last_q, split);

    float m[RW], l[RW], acc[RW][NE];
#pragma unroll
    for (int rr = 0; rr < RW; rr++) {
        m[rr] = -INFINITY;
        l[rr] = 0.f;
#pragma unroll
        for (int e = 0; e < NE; e++) acc[rr][e] = 0.f;
    }

    for (int ti = tiles.my_lo; ti < tiles.my_hi; ti++) {
        const int t = tiles.tile(ti);
        __syncthreads();
        // each warp stages 8 keys of the tile
        for (int jj = 0; jj < 8; jj++) {
            int j = warp * 8 + jj;
            int key = t * KT + j;
            if (key <= hi_pos) {
                int64_t page = page_of(bt, key, p.bt_stride, p.pages);
                int64_t at = (page * p.kv_heads + kvh) * GB_PAGE + (key % GB_PAGE);
                const T* kp = (const T*)p.k_plane + at * (int64_t)d;
                const T* vp = (const T*)p.v_plane + (vh < 0 ? at : (page * v_heads + vh) * GB_PAGE + (key % GB_PAGE)) * v_tok;
                for (int c = lane; c < d; c += 32) Ks[j * ks + c] = to_f32<T>(kp[c]);
                for (int c = lane; c < dv; c += 32) Vs[j * vs + c] = to_f32<T>(vp[c]);
            } else {
                for (int c = lane; c < d; c += 32) Ks[j * ks + c] = 0.f;
                for (int c = lane; c < dv; c += 32) Vs[j * vs + c] = 0.f;
            }
        }
        __syncthreads();

        float s[RW];
#pragma unroll
        for (int rr = 0; rr < RW; rr++) s[rr] = 0.f;
        const float* krow = Ks + lane * ks;
        const float* qrow = Qs + warp * RW * d;
        for (int c = 0; c < d; c++) {
            float kv = krow[c];
#pragma unroll
            for (int rr = 0; rr < RW; rr++) s[rr] = fmaf(qrow[rr * d + c], kv, s[rr]);
        }
        const int key = t * KT + lane;
        float pr[RW];
#pragma unroll
        for (int rr = 0; rr < RW; rr++) pr[rr] = weigh(row_ok[rr] && sees(p, row_pos[rr], key), s[rr], m[rr], l[rr], acc[rr]);
        for (int jj = 0; jj < KT; jj++) {
            const float* vrow = Vs + jj * vs;
#pragma unroll
            for (int rr = 0; rr < RW; rr++) {
                float pj = __shfl_sync(0xffffffffu, pr[rr], jj);
#pragma unroll
                for (int e = 0; e < NE; e++) {
                    int c = lane + 32 * e;
                    if (c < dv) acc[rr][e] = fmaf(pj, vrow[c], acc[rr][e]);
                }
            }
        }
    }

#pragma unroll
    for (int rr = 0; rr < RW; rr++)
        if (row_ok[rr]) leave_row<T>(p, seq, split, q_start + row_q[rr], row_head[rr], dv, lane, m[rr], l[rr], acc[rr]);
}

// The same for float32 rows of 16-byte chunks (the true 32-bit path at the usual head sizes), with the
// same additions in the same order.  The kernel above is bound by latency: it waits for every tile, key
// by key, before it computes on it, and a single token leaves all but one of its warps idle.  Here the next
// tile is on its way while one is worked on (cp.async, one page lookup a tile, two stages where they
// fit), keys, queries and probabilities are read four at a time, and a warp holds RW rows: one
// where a sequence brings at most four (the heads of a single token), so that its rows share out over
// the warps.
// Measured in the 32-bit steps of the 1.7B sizes (16 heads over 8 of 128): single tokens of three sequences of up to 333 keys
// 210 -> 35 us, two prompts of 201 and 140 tokens 113 -> 46 us.
template <int NE, int RW>
__global__ void __launch_bounds__(128) attn_f32_kernel(AttnParamsX p, int stages) {
    extern __shared__ __align__(16) float sm[];
    constexpr int ROWS = 4 * RW;
    const int d = p.d, ks = d + 4;
    const int dv = p.dv > 0 ? p.dv : p.d, vs = dv + 4;
    const int64_t v_tok = p.v_row_stride > 0 ? p.v_row_stride : dv;
    float* Qs = sm;                        // [ROWS][d], pre-scaled
    float* Ps = Qs + ROWS * d;             // [4 warps][RW][32]
    float* KV = Ps + ROWS * KT;            // [stages]: [32][d + 4], [32][dv + 4]
    const int stage_floats = KT * (ks + vs);

    const int G = p.heads / p.kv_heads;
    const int GC = G < ROWS ? G : ROWS;
    const int hchunks = (G + GC - 1) / GC;
    const int QT = ROWS / GC;

    const int seq = blockIdx.z / p.num_splits, split = blockIdx.z % p.num_splits;
    const int kvh = blockIdx.y / hchunks, chunk = blockIdx.y % hchunks;
    const int v_heads = p.v_share > 1 ? p.kv_heads / p.v_share : p.kv_heads, vh = p.v_share > 1 ? kvh / p.v_share : -1;
    const int q_len = p.seq_q_len[seq], kv_len = p.seq_kv_len[seq];
    const int q0 = (gridDim.x - 1 - blockIdx.x) * QT;  // late (long) tiles first
    if (q0 >= q_len) return;
    const int past = kv_len - q_len;
    const int q_start = p.seq_q_start[seq];
    const int* bt = block_table_row(p.block_table, p.bt_stride, p.seq_slot[seq], p.max_slots);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int last_q = (q0 + QT < q_len ? q0 + QT : q_len) - 1;
    const int hi_pos = past + last_q;
    const KeyTiles tiles(p, past, q0, last_q, split);
    const int my_lo = tiles.my_lo, my_hi = tiles.my_hi;

    // a tile's 32 keys lie in one page (of 64, and tiles begin at multiples of 32); its first key is visible
    auto load = [&](int ti) {
        const int t = tiles.tile(ti);
        const int64_t page = page_of(bt, t * KT, p.bt_stride, p.pages);
        const int64_t at = (page * p.kv_heads + kvh) * GB_PAGE + (t * KT) % GB_PAGE;
        const float* kp = (const float*)p.k_plane + at * d;
        const float* vp = (const float*)p.v_plane + (vh < 0 ? at : (page * v_heads + vh) * GB_PAGE + (t * KT) % GB_PAGE) * v_tok;
        float* K = KV + (ti - my_lo) % stages * stage_floats;
        float* V = K + KT * ks;
        const int rows = hi_pos + 1 - t * KT;  // keys of the tile that anyone sees; zeros behind them
        for (int i = tid; i < KT * (d / 4); i += 128) {
            const int j = i / (d / 4), c = (i - j * (d / 4)) * 4;
            cp_async16(K + j * ks + c, kp + (j < rows ? (int64_t)j * d + c : 0), j < rows ? 16 : 0);
        }
        for (int i = tid; i < KT * (dv / 4); i += 128) {
            const int j = i / (dv / 4), c = (i - j * (dv / 4)) * 4;
            cp_async16(V + j * vs + c, vp + (j < rows ? j * v_tok + c : 0), j < rows ? 16 : 0);
        }
    };
    for (int i = 0; i < stages - 1; i++) {
        if (my_lo + i < my_hi) load(my_lo + i);
        cp_async_commit();
    }

    for (int idx = tid; idx < ROWS * d; idx += 128) {
        int r = idx / d, c = idx - r * d;
        int qi = r / GC, hg = chunk * GC + r % GC;
        bool ok = qi < QT && q0 + qi < q_len && hg < G;
        float v = 0.f;
        if (ok) v = ((const float*)p.q)[(int64_t)(q_start + q0 + qi) * p.q_row_stride + (int64_t)(kvh * G + hg) * d + c] * p.scale;
        Qs[idx] = v;
    }
    int row_pos[RW], row_head[RW], row_q[RW];
    bool row_ok[RW], any = false;
#pragma unroll
    for (int rr = 0; rr < RW; rr++) {
        int r = warp * RW + rr;
        int qi = r / GC, hg = chunk * GC + r % GC;
        row_ok[rr] = qi < QT && q0 + qi < q_len && hg < G;
        any |= row_ok[rr];
        row_q[rr] = q0 + qi;
        row_head[rr] = kvh * G + hg;
        row_pos[rr] = past + q0 + qi;
    }

    float m[RW], l[RW], acc[RW][NE];
#pragma unroll
    for (int rr = 0; rr < RW; rr++) {
        m[rr] = -INFINITY;
        l[rr] = 0.f;
#pragma unroll
        for (int e = 0; e < NE; e++) acc[rr][e] = 0.f;
    }

    float* pw = Ps + warp * RW * KT;
    const float* qrow = Qs + warp * RW * d;
    for (int ti = my_lo; ti < my_hi; ti++) {
        const int t = tiles.tile(ti);
        if (stages == 1) {
            __syncthreads();  // all are done with the tile before
            load(ti);
            cp_async_commit();
        }
        cp_async_wait<0>();
        __syncthreads();      // the tile is visible to all; with two stages, all are done with the tile before as well
        if (stages == 2) {
            if (ti + 1 < my_hi) load(ti + 1);
            cp_async_commit();
        }
        if (!any) continue;   // no row of this warp: it only helps to fetch
        const float* K = KV + (ti - my_lo) % stages * stage_floats;
        const float* V = K + KT * ks;

        float s[RW];
#pragma unroll
        for (int rr = 0; rr < RW; rr++) s[rr] = 0.f;
        const float* krow = K + lane * ks;
#pragma unroll 4
        for (int c = 0; c < d; c += 4) {
            const float4 kv = *(const float4*)(krow + c);
#pragma unroll
            for (int rr = 0; rr < RW; rr++) {
                const float4 qv = *(const float4*)(qrow + rr * d + c);
                s[rr] = fmaf(qv.x, kv.x, s[rr]);
                s[rr] = fmaf(qv.y, kv.y, s[rr]);
                s[rr] = fmaf(qv.z, kv.z, s[rr]);
                s[rr] = fmaf(qv.w, kv.w, s[rr]);
            }
        }
        const int key = t * KT + lane;
        __syncwarp();         // the probabilities of the tile before have been read
#pragma unroll
        for (int rr = 0; rr < RW; rr++)
            pw[rr * KT + lane] = weigh(row_ok[rr] && sees(p, row_pos[rr], key), s[rr], m[rr], l[rr], acc[rr]);
        __syncwarp();
#pragma unroll 2
        for (int j0 = 0; j0 < KT; j0 += 4) {
            float pr[RW][4];
#pragma unroll
            for (int rr = 0; rr < RW; rr++) *(float4*)pr[rr] = *(const float4*)(pw + rr * KT + j0);
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const float* vrow = V + (j0 + jj) * vs;
#pragma unroll
                for (int e = 0; e < NE; e++) {
                    const int c = lane + 32 * e;
                    if (c < dv) {
                        const float v = vrow[c];
#pragma unroll
                        for (int rr = 0; rr < RW; rr++) acc[rr][e] = fmaf(pr[rr][jj], v, acc[rr][e]);
                    }
                }
            }
        }
    }
    cp_async_wait<0>();

#pragma unroll
    for (int rr = 0; rr < RW; rr++)
        if (row_ok[rr]) leave_row<float>(p, seq, split, q_start + row_q[rr], row_head[rr], dv, lane, m[rr], l[rr], acc[rr]);
}

// out[seq, head, :] = sum_s exp(m_s - M) acc_s / sum_s exp(m_s - M) l_s over the key splits, one CTA a (sequence, head) and a
// thread a value.  Every warp finds the maximum, the normaliser and the weights for itself (a lane a split, shuffle trees, a fixed
// order); thread c then adds value c of the splits in split order.  A chain of waits for memory and little else, so what it
// reads is asked for at once: the first splits' values beside all maxima and sums (one behind the other, with the weights
// through shared memory, and so; attention and merge in a chain, us: one sequence of 4096 keys, 32 heads of 128 in 16 splits 13.4
// and 11.6, one of 4096 latents in 16 splits 28.0 and 21.9, 24 of 1500 in 5 splits 30.1 and 25.8).
constexpr int MERGE_MAX_SPLITS = 256;
constexpr int MERGE_THREADS = 512;
constexpr int MERGE_AHEAD = 8;    // splits whose values are asked for ahead

template <typename T>
__global__ void __launch_bounds__(MERGE_THREADS) attn_merge_kernel(AttnParamsX p, int d) {
    pdl_trigger();  // the product that follows may start fetching its weights
    const int head = blockIdx.x, seq = blockIdx.y, lane = threadIdx.x & 31, c = threadIdx.x;
    const float* sp = p.scratch + ((int64_t)seq * p.heads + head) * p.num_splits * (d + 2);
    const float* column = sp + 2 + (c < d ? c : 0);
    const int n = p.num_splits;
    const float m = lane < n ? sp[(int64_t)lane * (d + 2)] : -INFINITY, l = lane < n ? sp[(int64_t)lane * (d + 2) + 1] : 0.f;
    float v[MERGE_AHEAD];
#pragma unroll
    for (int j = 0; j < MERGE_AHEAD; j++) v[j] = j < n ? column[(int64_t)j * (d + 2)] : 0.f;
    float M = m;
    for (int s = lane + 32; s < n; s += 32) M = fmaxf(M, sp[(int64_t)s * (d + 2)]);
    M = warp_max(M);
    const float z = p.sinks ? p.sinks[head] : 0.f;  // the sink's score
    if (p.sink) M = fmaxf(M, z);
    const float w0 = m != -INFINITY ? expf(m - M) : 0.f;
    float L = lane < n ? w0 * l : 0.f;
    for (int s = lane + 32; s < n; s += 32) {
        const float ms = sp[(int64_t)s * (d + 2)];
        L += (ms != -INFINITY ? expf(ms - M) : 0.f) * sp[(int64_t)s * (d + 2) + 1];
    }
    L = warp_sum(L);
    if (p.sink) L += expf(z - M);
    float a = 0.f;
    for (int s0 = 0; s0 < n; s0 += 32) {
        float w = w0;
        if (s0 > 0) {
            const float ms = s0 + lane < n ? sp[(int64_t)(s0 + lane) * (d + 2)] : -INFINITY;
            w = ms != -INFINITY ? expf(ms - M) : 0.f;
        }
        for (int s1 = s0; s1 < n && s1 < s0 + 32; s1 += MERGE_AHEAD) {
            if (s1 > 0) {
#pragma unroll
                for (int j = 0; j < MERGE_AHEAD; j++) v[j] = s1 + j < n ? column[(int64_t)(s1 + j) * (d + 2)] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < MERGE_AHEAD; j++) {
                const float wj = __shfl_sync(0xffffffffu, w, s1 - s0 + j);
                if (s1 + j < n) a += wj * v[j];
            }
        }
    }
    if (c < d) ((T*)p.out)[(int64_t)p.seq_q_start[seq] * p.out_row_stride + (int64_t)head * d + c] = from_f32<T>(a / L);
}

// a thread a value where there are that many (four rounds of loads one behind the other for heads of 512 took 6 us)
int merge_threads(int dv) { return dv <= 128 ? 128 : dv < MERGE_THREADS ? (dv + 31) / 32 * 32 : MERGE_THREADS; }

template <typename T, int NE>
int launch_ne(const AttnParamsX& p, dim3 grid, size_t smem, cudaStream_t stream) {
    static bool configured = false;
    if (!configured && smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(attn_simt_kernel<T, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (e != cudaSuccess) GB_REFUSE("attention_simt: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    attn_simt_kernel<T, NE><<<grid, 128, smem, stream>>>(p);
    GB_CHECK_LAUNCH("attention_simt");
    return 0;
}

// float32 operands whose rows are 16-byte chunks
bool chunked_f32(const AttnParamsX& p) {
    const int dv = p.dv > 0 ? p.dv : p.d;
    return (p.d & 3) == 0 && (dv & 3) == 0 && (p.v_row_stride & 3) == 0 && !((uintptr_t)p.k_plane & 15) && !((uintptr_t)p.v_plane & 15);
}

template <int NE, int RW>
int launch_f32_ne(const AttnParamsX& p, cudaStream_t stream) {
    constexpr int ROWS = 4 * RW;
    const int G = p.heads / p.kv_heads, GC = G < ROWS ? G : ROWS, dv = p.dv > 0 ? p.dv : p.d;
    const dim3 grid(ceil_div(p.max_q_len, ROWS / GC), p.kv_heads * ceil_div(G, GC), p.nseq * p.num_splits);
    if (grid.y > 65535 || grid.z > 65535) GB_REFUSE("attention_simt: grid (%u, %u, %u) exceeds one launch", grid.x, grid.y, grid.z);
    const size_t fixed = (size_t)ROWS * (p.d + KT) * 4, stage = (size_t)KT * (p.d + dv + 8) * 4;
    const int stages = fixed + 2 * stage <= 110 * 1024 ? 2 : 1;  // two stages only where two CTAs still fit an SM
    static bool configured[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) GB_REFUSE("attention_simt: no current device");
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attn_f32_kernel<NE, RW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (e != cudaSuccess) GB_REFUSE("attention_simt: cannot reserve shared memory: %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    attn_f32_kernel<NE, RW><<<grid, 128, fixed + stages * stage, stream>>>(p, stages);
    GB_CHECK_LAUNCH("attention_simt");
    return 0;
}

int launch_f32(const AttnParamsX& p, cudaStream_t stream) {
    const int G = p.heads / p.kv_heads, dv = p.dv > 0 ? p.dv : p.d;
    const bool few = (int64_t)p.max_q_len * G <= 4;
    switch (ceil_div(dv, 32)) {
        case 1: return few ? launch_f32_ne<1, 1>(p, stream) : launch_f32_ne<1, 4>(p, stream);
        case 2: return few ? launch_f32_ne<2, 1>(p, stream) : launch_f32_ne<2, 4>(p, stream);
        case 3: case 4: return few ? launch_f32_ne<4, 1>(p, stream) : launch_f32_ne<4, 4>(p, stream);
        case 5: case 6: case 7: case 8: return few ? launch_f32_ne<8, 1>(p, stream) : launch_f32_ne<8, 4>(p, stream);
        default: return few ? launch_f32_ne<16, 1>(p, stream) : launch_f32_ne<16, 4>(p, stream);
    }
}

template <typename T>
int launch(const AttnParamsX& p, cudaStream_t stream) {
    const int G = p.heads / p.kv_heads;
    const int GC = G < ROWS ? G : ROWS;
    const int hchunks = (G + GC - 1) / GC;
    const int QT = ROWS / GC;
    dim3 grid(ceil_div(p.max_q_len, QT), p.kv_heads * hchunks, p.nseq * p.num_splits);
    if (grid.y > 65535 || grid.z > 65535)
        GB_REFUSE("attention_simt: grid (%u, %u, %u) exceeds one launch", grid.x, grid.y, grid.z);
    const int dv = p.dv > 0 ? p.dv : p.d;
    size_t smem = ((size_t)ROWS * p.d + (size_t)KT * (p.d + 1) + (size_t)KT * (dv + 1)) * sizeof(float);
    int ne = ceil_div(dv, 32);
    int rc;
    if (std::is_same<T, float>::value && chunked_f32(p))
        rc = launch_f32(p, stream);
    else switch (ne) {
        case 1: rc = launch_ne<T, 1>(p, grid, smem, stream); break;
        case 2: rc = launch_ne<T, 2>(p, grid, smem, stream); break;
        case 3: rc = launch_ne<T, 3>(p, grid, smem, stream); break;
        case 4: rc = launch_ne<T, 4>(p, grid, smem, stream); break;
        case 5: rc = launch_ne<T, 5>(p, grid, smem, stream); break;
        case 6: rc = launch_ne<T, 6>(p, grid, smem, stream); break;
        case 7: rc = launch_ne<T, 7>(p, grid, smem, stream); break;
        case 8: rc = launch_ne<T, 8>(p, grid, smem, stream); break;
        case 9: case 10: case 11: case 12: rc = launch_ne<T, 12>(p, grid, smem, stream); break;
        case 13: case 14: case 15: case 16: rc = launch_ne<T, 16>(p, grid, smem, stream); break;
        default: GB_REFUSE("attention_simt: value size %d is larger than %d", dv, SIMT_MAX_DV);
    }
    if (rc) return rc;
    if (p.num_splits > 1) {
        attn_merge_kernel<T><<<dim3(p.heads, p.nseq), merge_threads(dv), 0, stream>>>(p, dv);
        GB_CHECK_LAUNCH("attention_merge");
    }
    return 0;
}

}  // namespace

// Merge of per-split partial results, shared with the tensor-core single-token kernel.
int gb_attention_merge_launch(const AttnParamsX& p, int dv, int dtype, cudaStream_t stream) {
    if (p.num_splits > MERGE_MAX_SPLITS) GB_REFUSE("attention: %d key splits; at most %d", p.num_splits, MERGE_MAX_SPLITS);
    if (dtype == GB_F32)
        attn_merge_kernel<float><<<dim3(p.heads, p.nseq), merge_threads(dv), 0, stream>>>(p, dv);
    else
        attn_merge_kernel<__nv_bfloat16><<<dim3(p.heads, p.nseq), merge_threads(dv), 0, stream>>>(p, dv);
    GB_CHECK_LAUNCH("attention_merge");
    return 0;
}

GB_API int gb_attention_simt(const AttnParams* pp, int dtype, cudaStream_t stream) {
    const AttnParamsX x = gb_attn_widen(*pp);
    return gb_attention_simt_x(&x, dtype, stream);
}

GB_API int gb_attention_simt_x(const AttnParamsX* pp, int dtype, cudaStream_t stream) {
    AttnParamsX p = *pp;
    if (p.nseq <= 0 || p.max_q_len <= 0) return 0;
    if (p.heads <= 0 || p.kv_heads <= 0 || p.heads % p.kv_heads) GB_REFUSE("attention: %d heads over %d kv heads", p.heads, p.kv_heads);
    if (p.d <= 0 || p.d > SIMT_MAX_D) GB_REFUSE("attention_simt: head_dim %d is outside [1, %d]", p.d, SIMT_MAX_D);
    if (p.num_splits < 1 || p.num_splits > MERGE_MAX_SPLITS) GB_REFUSE("attention: %d key splits; 1 to %d", p.num_splits, MERGE_MAX_SPLITS);
    if (p.num_splits > 1 && p.max_q_len != 1) GB_REFUSE("attention: key splits need single-token rows, got rows of up to %d", p.max_q_len);
    if (p.num_splits > 1 && !p.scratch) GB_REFUSE("attention: %d key splits without scratch memory", p.num_splits);
    if (p.window < 0) GB_REFUSE("attention: window %d", p.window);
    if (p.dv < 0 || p.dv > SIMT_MAX_DV || (p.dv == 0 && p.d > SIMT_MAX_DV)) GB_REFUSE("attention_simt: value size %d is outside [1, %d]", p.dv ? p.dv : p.d, SIMT_MAX_DV);
    if (p.chunk < 0) GB_REFUSE("attention: blocks of %d positions", p.chunk);
    if (p.v_share < 0 || (p.v_share > 1 && p.kv_heads % p.v_share)) GB_REFUSE("attention: %d key heads share value heads by %d", p.kv_heads, p.v_share);
    if (p.v_row_stride < 0 || (p.v_row_stride > 0 && p.v_row_stride < (p.dv ? p.dv : p.d))) GB_REFUSE("attention: value stride %lld", (long long)p.v_row_stride);
    if (p.keep_first < 0) GB_REFUSE("attention: %d kept first tokens", p.keep_first);
    if (dtype == GB_F32) return launch<float>(p, stream);
    if (dtype == GB_BF16) return launch<__nv_bfloat16>(p, stream);
    GB_REFUSE("attention: unknown dtype %d", dtype);
}

// the checked build's record of the first index this file's kernels found out of bounds
GB_CHECK_READER(gb_checked_status_attention_simt)
