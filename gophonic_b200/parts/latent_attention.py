"""Latent attention over the paged cache (``LatentAttentionSpec``): queries, keys and values are made from low-rank
latents and only the key/value latent c and one rotated key part k_r are cached, kv_rank + rot_dim numbers a token.

How it runs.  A head's plain key is W_uk c and its value W_uv c, so a score is q_plain . (W_uk c) + q_rot . k_r =
(W_uk^T q_plain) . c + q_rot . k_r and a head's output is W_uv (sum_j p_j c_j): the products with W_uk and W_uv move
from the keys to the queries and to the outputs, and attention itself runs over the cache as it is, as one key head of
kv_rank + rot_dim channels that all query heads read and whose first kv_rank channels are also the values (the
cache keeps no value plane: ``KVRequest.values_in_keys``).  Nothing is expanded per cached token, so prompts in
portions, single tokens and batches are one path.  A prompt whose rows see the same keys many times over takes the other
order in bfloat16: the latents that the step can see are gathered (``ops.latent_gather``), expanded to keys and values of every
head by two products and attended to as such on the tcgen05 kernel (``ops.attention_latent_expanded``), three and a
half times fewer operations a pair; the cache is the same.

Per step: one product for both down-projections (and the output gate's pre-activations, if there is one); a row-wise kernel for the two RMS norms, the rotation of k_r and the
cache write (``ops.latent_prep``); the query up-projection; the per-head product with W_uk and the rotation of the
queries' rotated part into the absorbed queries; attention; the per-head product with W_uv; the output projection.
The per-head products are one launch for all heads: on the tensor cores (mma.sync) in bfloat16, on the CUDA cores in float32
and for few rows that kernel cannot take; what neither takes runs one product a head.
"""
from __future__ import annotations

from typing import List, Mapping

import torch

from .. import registry
from .attention import choose_splits, page_class
from .base import KVRequest, Mixer, Runtime, TensorDecl


class LatentAttention(Mixer):
    capturable = True
    EXPANDED_KEYS_A_ROW, EXPANDED_BYTES, FEW_ROWS_PAGES = 12, 128 << 20, 20
    ROWS_ONE_LAUNCH = 32      # up to this many rows the per-head products that the tensor cores do not take run as one launch

    @classmethod
    def declare(cls, spec, prefix: str) -> List[TensorDecl]:
        n = dict(spec.names)
        H, d, dr, dv, Q, R = spec.heads, spec.head_dim, spec.rot_dim, spec.value_dim, spec.q_rank, spec.kv_rank
        return [TensorDecl(prefix + n["dq"], (Q, spec.hidden)), TensorDecl(prefix + n["dq_norm"], (Q,), role="norm"),
                TensorDecl(prefix + n["uq"], (H * (d + dr), Q)), TensorDecl(prefix + n["dkv"], (R + dr, spec.hidden)),
                TensorDecl(prefix + n["dkv_norm"], (R,), role="norm"), TensorDecl(prefix + n["uk"], (H * d, R)),
                TensorDecl(prefix + n["uv"], (H * dv, R))] + (
                    [TensorDecl(prefix + n["g"], (H * dv, spec.hidden))] if getattr(spec, "gate", False) else []) + [
                TensorDecl(prefix + n["o"], (spec.hidden, H * dv))]

    @classmethod
    def cache_request(cls, spec):
        return KVRequest(kv_heads=1, head_dim=spec.kv_rank + spec.rot_dim, window=0, value_dim=spec.kv_rank, values_in_keys=True)

    def __init__(self, spec, prefix: str, tensors: Mapping[str, torch.Tensor], runtime: Runtime):
        self.spec, self.rt = spec, runtime
        n = dict(spec.names)
        H, d, dv, R = spec.heads, spec.head_dim, spec.value_dim, spec.kv_rank
        dq, dkv = tensors[prefix + n["dq"]], tensors[prefix + n["dkv"]]
        if dq.dtype != dkv.dtype:
            raise ValueError(f"{prefix}: the down-projections are stored as {dq.dtype} and {dkv.dtype}; they must agree")
        parts = [dq, dkv]
        self.gated = bool(getattr(spec, "gate", False))
        if self.gated:
            parts.append(tensors[prefix + n["g"]])
            if parts[2].dtype != dq.dtype:
                raise ValueError(f"{prefix}: the down-projections are {dq.dtype} and the gate's matrix {parts[2].dtype}; they must agree")
        self.down = torch.cat(parts, dim=0).contiguous()              # x is read once
        self.uq = tensors[prefix + n["uq"]].contiguous()
        uk, uv = tensors[prefix + n["uk"]], tensors[prefix + n["uv"]]
        # a head's W_uk is [head_dim, kv_rank]: as stored it maps plain query channels (K) to latent channels (N)
        self.uk_kn = uk.view(H, d, R).contiguous()
        self.uk_nk = self.uk_kn.transpose(1, 2).contiguous()          # [heads, kv_rank, head_dim] for a product a head
        self.uv_nk = uv.view(H, dv, R).contiguous()                   # as stored: latent channels (K) to value channels (N)
        self.uv_kn = self.uv_nk.transpose(1, 2).contiguous()
        self.o = tensors[prefix + n["o"]].contiguous()
        self.q_norm = tensors[prefix + n["dq_norm"]].to(torch.float32).contiguous()
        self.kv_norm = tensors[prefix + n["dkv_norm"]].to(torch.float32).contiguous()
        self.position = registry.part_class("position", spec.position.kind)(spec.position, prefix, tensors, runtime)
        if spec.rot_dim > 0 and not getattr(self.position, "pairs", False):
            raise ValueError(f"{prefix}: the rotated key part turns neighbouring channels together; position kind '{spec.position.kind}' does not")
        self.key_dim = R + spec.rot_dim

    def weight_bytes(self) -> int:
        ts = (self.down, self.uq, self.uk_kn, self.uv_nk, self.o)
        return sum(t.numel() * t.element_size() for t in ts)

    def prepare(self, capacity: int) -> None:
        self.position.prepare(capacity)

    def plan(self, nseq: int, max_q_len: int, max_kv_len: int, sm_count: int):
        if max_q_len != 1:
            return 1
        s = self.spec
        seen = max_kv_len
        for size in (s.chunk, s.window):
            if size > 0:
                seen = min(seen, size)
        elem = 4 if self.rt.is_fp32 else 2
        # a page of latents fills most of an SM's shared memory twice over: one CTA an SM, where the model of the split
        # choice counts two
        splits = choose_splits(nseq, seen, max(1, sm_count // 2), 64 * self.key_dim * elem)
        return splits if self.rt.is_fp32 else max(splits, self.fine_splits(nseq, seen, sm_count))

    def fine_splits(self, nseq: int, seen: int, sm_count: int) -> int:
        """Into how many pieces at least single tokens in bfloat16 are cut: as many as run in one wave of an SM a CTA, down to a page each,
        where that pays.  A page takes a CTA 3.3 us at a latent of 512, and the merge about as long as two, and as one more for every 12
        sequences of 16 heads (whole steps of eight layers, six of them over latents, against ``choose_splits`` alone: 4 sequences of
        250 keys -4 %, 4 of 700 -11, 16 of 350 -3, 24 of 700 -6; without the last condition 16 of 250 +3, 48 of 350 +3, 64 of
        700 +1).  Narrower latents leave room for more CTAs an SM and keep to ``choose_splits``."""
        s = self.spec
        most = min(32, sm_count // max(1, nseq * -(-s.heads // 32)))     # a CTA holds up to 32 heads
        if most < 2 or s.kv_rank != 512 or self.key_dim % 16 or self.key_dim > 640:
            return 1
        pages = (seen + 63) // 64
        size = page_class(pages)
        splits = -(-size // -(-size // most))
        saved = pages - -(-pages // splits)
        return splits if 192 * (saved - 2) > nseq * s.heads else 1

    def key_splits(self, batch):
        s = self.spec
        splits = int(batch.plan_for(self) or 1)
        if splits <= 1:
            return 1, None
        return splits, batch.workspace(("attention key splits", s.heads, s.kv_rank, splits),
                                       self.rt.ops.attention_scratch_floats(batch.nseq, s.heads, s.kv_rank, splits))

    def _per_head(self, a: torch.Tensor, w_kn: torch.Tensor, w_nk: torch.Tensor, out: torch.Tensor) -> None:
        """out[:, h, :] = a[:, h, :] @ w_kn[h] for every head (``w_nk`` holds the same matrices transposed)."""
        ops = self.rt.ops
        rows, heads, K = a.shape
        # bfloat16: the tensor cores from one row on (16 heads, us inside a graph: 128 x 512 one row 3.3 on the CUDA cores and 2.4, 24
        # rows 7.3 and 2.6; 512 x 128 7.4 and 5.6, 24 rows 11.4 and 5.8; as many outputs are the nearest to the 64-bit sum)
        if ops.head_gemm_mma_accepts(a, w_nk, out):
            ops.head_gemm_mma(a, w_nk, out)
            return
        if (self.rt.is_fp32 or rows <= self.ROWS_ONE_LAUNCH) and K <= ops.HEAD_GEMM_MAX_K:
            ops.head_gemm(a, w_kn, out)
            return
        for h in range(heads):
            ops.gemm(a[:, h, :], w_nk[h], out[:, h, :])

    def runs(self, batch):
        """The step's sequences in neighbouring runs (first sequence, end, first row, end, most rows of one, pages): ``pages`` of the
        cache are what the run's rows see if it goes over expanded keys and values, 0 if over the latents.

        Over the latents a (row, key) pair of a head costs kv_rank + rot_dim + kv_rank multiply-adds, over expanded keys and
        values head_dim + rot_dim + value_dim (1088 against 320 at a latent of 512), and the expansion itself
        kv_rank (head_dim + value_dim) a key.  So it pays where a key is seen by enough rows.  Measured over eight layers (16
        heads, a latent of 512, a window of 1024; ms a step, absorbed and expanded): 3244 rows over 3264 keys 8.4 and 4.9,
        3741 over 12160 11.1 and 5.9, 1121 over 9280 6.3 and 3.4; 128 over 1152 and 70 over 1088 the same, 261 rows of
        four sequences over 4352 3.5 and 3.6.

        Both forms round, at different places, so a sequence's form must not follow from the other sequences' contexts: the numbers of
        sequences and rows, by which all kernels are chosen, decide for the step.  A key of a sequence is seen by as many rows as
        the portion and the window have, so what counts is the mean portion: with a window so many rows that at most twelve
        keys a row are visible, without one the 94 rows that a window of 1024 asks for.

        A run of its own costs the host about 0.1 ms a layer (eight layers, us: 300, 9, 120 and 1 row behind 300 tokens 2855 in one
        run, 4650 in four), so a sequence leaves the others' form only for its own sake: few rows behind so many keys that the
        expansion costs more than that.  The expanded rows are scratch memory, no more of it at a time than the absorbed queries and
        outputs of the same sequences would take, or EXPANDED_BYTES; a run that would is cut in two, a sequence that would
        alone stays on the latents."""
        s = self.spec
        key = ("latent runs", s.heads, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank, s.window, self.uk_kn.dtype, self.uv_nk.dtype)
        if key not in batch.shared:       # every layer of one geometry has the same answer
            batch.shared[key] = self._runs(batch)
        return batch.shared[key]

    def _runs(self, batch):
        s, ops = self.spec, self.rt.ops
        window = int(s.window)
        if (batch.extents is None or not ops.latent_expanded_accepts(self.rt.act_dtype, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank, batch.max_q_len)
                or self.uk_kn.dtype != torch.bfloat16 or self.uv_nk.dtype != torch.bfloat16
                or batch.nseq * (window if window > 0 else 1024) > (self.EXPANDED_KEYS_A_ROW - 1) * batch.rows):
            return [(0, batch.nseq, 0, batch.rows, batch.max_q_len, 0)]
        page_bytes = 2 * 64 * (self.key_dim + s.heads * (s.head_dim + s.value_dim))
        row_bytes = 2 * s.heads * (self.key_dim + s.kv_rank)
        out, at = [], 0
        for i, (known, rows) in enumerate(batch.extents):
            pages = (known + rows + 63) // 64 - (max(0, known - window + 1) // 64 if window > 0 else 0)
            if (rows < ops.LATENT_TC5_MIN_ROWS and pages > self.FEW_ROWS_PAGES) or pages * page_bytes > max(rows * row_bytes, self.EXPANDED_BYTES):
                pages = 0
            if out and (out[-1][5] > 0) == (pages > 0):
                first, _, lo, _, most, held = out[-1]
                if not pages or (held + pages) * page_bytes <= max((at + rows - lo) * row_bytes, self.EXPANDED_BYTES):
                    out[-1] = (first, i + 1, lo, at + rows, max(most, rows), held + pages)
                    at += rows
                    continue
            out.append((i, i + 1, at, at + rows, rows, pages))
            at += rows
        return out

    @staticmethod
    def _sequences(batch, run):
        """(slots, first rows, rows, keys) of the run's sequences and the positions of its rows."""
        first, end, lo, hi = run[:4]
        if end - first == batch.nseq:
            return batch.seq_slot, batch.seq_q_start, batch.seq_q_len, batch.seq_kv_len, batch.row_pos
        return batch.seq_slot[first:end], batch.seq_q_start[first:end], batch.seq_q_len[first:end], batch.seq_kv_len[first:end], batch.row_pos[lo:hi]

    def _expanded(self, batch, q: torch.Tensor, ctx: torch.Tensor, cache, run) -> None:
        """Attention of a run's rows over keys and values made from the visible latents for this step."""
        ops, s = self.rt.ops, self.spec
        H, R, dev = s.heads, s.kv_rank, q.device
        first, end, lo, hi, most, pages = run
        slot, q_start, q_len, kv_len, row_pos = self._sequences(batch, run)
        cos, sin, _ = self.position.kernel_args()
        mine = q if hi - lo == batch.rows else q[lo:hi]
        ops.latent_q_rot(mine, mine, H, s.head_dim, s.rot_dim, cos, sin, row_pos)
        lat = torch.empty((64 * pages, self.key_dim), dtype=q.dtype, device=dev)
        base = torch.empty((end - first,), dtype=torch.int32, device=dev)
        ops.latent_gather(cache.k, cache.block_table, slot, q_len, kv_len, end - first, int(s.window), lat, base)
        keys = torch.empty((64 * pages, H * s.head_dim), dtype=q.dtype, device=dev)
        values = torch.empty((64 * pages, H * s.value_dim), dtype=q.dtype, device=dev)
        ops.gemm(lat[:, :R], self.uk_kn.view(H * s.head_dim, R), keys)
        ops.gemm(lat[:, :R], self.uv_nk.view(H * s.value_dim, R), values)
        ops.attention_latent_expanded(q, ctx, keys, values, lat, base, R, q_start, q_len, kv_len, end - first, most, H, float(s.scale),
                                      int(s.window), int(s.chunk))

    def _absorbed(self, batch, q: torch.Tensor, ctx: torch.Tensor, cache, run) -> None:
        """Attention of a run's rows over the latents as they are cached."""
        ops, s = self.rt.ops, self.spec
        H, d, dr, dv, R = s.heads, s.head_dim, s.rot_dim, s.value_dim, s.kv_rank
        first, end, lo, hi, most, _ = run
        slot, q_start, q_len, kv_len, row_pos = self._sequences(batch, run)
        rows = hi - lo
        if rows != batch.rows:
            q, ctx, q_start = q[lo:hi], ctx[lo:hi], q_start - lo     # rows of qa
        cos, sin, _ = self.position.kernel_args()
        qa = torch.empty((rows, H * self.key_dim), dtype=q.dtype, device=q.device)       # per head [W_uk^T q_plain | rotated part]
        self._per_head(q.view(rows, H, d + dr)[:, :, :d], self.uk_kn, self.uk_nk, qa.view(rows, H, self.key_dim)[:, :, :R])
        ops.latent_q_rot(q, qa, H, d, dr, cos, sin, row_pos)
        mixed = torch.empty((rows, H * R), dtype=q.dtype, device=q.device)               # per head sum_j p_j c_j
        splits, scratch = self.key_splits(batch)
        ops.attention(qa, mixed, cache.k, cache.v, cache.block_table, slot, q_start, q_len, kv_len, end - first, most, H, 1, self.key_dim,
                      float(s.scale), int(s.window), splits, scratch, value_dim=R, chunk=int(s.chunk))
        self._per_head(mixed.view(rows, H, R), self.uv_kn, self.uv_nk, ctx.view(rows, H, dv))

    def forward(self, batch, x: torch.Tensor, out: torch.Tensor, cache) -> None:
        ops, s = self.rt.ops, self.spec
        rows = x.shape[0]
        H, d, dr, dv, Q, R = s.heads, s.head_dim, s.rot_dim, s.value_dim, s.q_rank, s.kv_rank
        if cache is None:
            raise ValueError("attention needs a key/value cache plane")
        if cache.k.dtype != x.dtype:
            raise ValueError(f"attention: cache holds {cache.k.dtype}, activations are {x.dtype}")
        made = torch.empty((rows, self.down.shape[0]), dtype=x.dtype, device=x.device)   # [query latent | kv latent | k_r | gate]
        ops.gemm(x, self.down, made)
        lat = made[:, :Q + R + dr]
        cos, sin, _ = self.position.kernel_args()
        cq = torch.empty((rows, Q), dtype=x.dtype, device=x.device)
        ops.latent_prep(lat, cq, self.q_norm, self.kv_norm, float(s.eps), cos, sin, Q, R, dr, batch.row_pos, batch.row_seq, batch.seq_slot,
                        cache.block_table, cache.k, cache.writable)
        q = torch.empty((rows, H * (d + dr)), dtype=x.dtype, device=x.device)
        ops.gemm(cq, self.uq, q)
        ctx = torch.empty((rows, H * dv), dtype=x.dtype, device=x.device)
        for run in self.runs(batch):
            (self._expanded if run[5] else self._absorbed)(batch, q, ctx, cache, run)
        if self.gated:
            ops.head_norm_gate(ctx, made[:, Q + R + dr:], ctx, H, dv, ops.GATE_SIGMOID)
        ops.gemm(ctx, self.o, out)
