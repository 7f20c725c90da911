// Which keys a single token sees, as a list of cache pages, and into how many pieces that list is cut when every sequence is
// cut by its own length: what the attention kernels and the kernel that merges their pieces must agree on.
#pragma once

#include "api.h"
#include "common.cuh"

// The pages of the keys [0, keep_first) first, where a window leaves them visible, then those of [lo_pos, pos].
struct DecodeSpan {
    int pos, lo_pos, t_lo, n_first, n_tiles;
    __device__ __forceinline__ int tile_of(int i) const { return i < n_first ? i : t_lo + (i - n_first); }
};

__device__ __forceinline__ DecodeSpan attn_decode_span(const AttnParamsX& p, int pos) {
    DecodeSpan s;
    s.pos = pos;
    s.lo_pos = 0;
    if (p.window > 0) {
        s.lo_pos = pos - p.window + 1;
        if (s.lo_pos < 0) s.lo_pos = 0;
    }
    if (p.chunk > 0 && pos - pos % p.chunk > s.lo_pos) s.lo_pos = pos - pos % p.chunk;   // blocks of positions
    s.t_lo = s.lo_pos / GB_PAGE;
    s.n_first = p.window > 0 && p.keep_first > 0 ? (p.keep_first + GB_PAGE - 1) / GB_PAGE : 0;
    if (s.n_first > s.t_lo) s.n_first = s.t_lo;
    s.n_tiles = s.n_first + pos / GB_PAGE + 1 - s.t_lo;
    return s;
}

// Pieces of `piece_tiles` pages, or of as many more as it takes to need no more than `most`: a function of the sequence's own
// length, so that a sequence's sums do not depend on the others in its step.
__device__ __forceinline__ int attn_pieces(int n_tiles, int piece_tiles, int most) {
    const int least = (n_tiles + most - 1) / most;
    const int per = least > piece_tiles ? least : piece_tiles;
    return n_tiles > per ? (n_tiles + per - 1) / per : 1;
}
