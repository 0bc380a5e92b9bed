"""Sequence <-> head re-sharding for sequence-parallel attention (the "Ulysses" exchange), on top of the
uniform all-to-all.

Every rank holds a slice of the sequence with all heads, ``[S / P, H, D]``; attention wants the whole sequence
for a slice of the heads, ``[S, H / P, D]``.  Going there and back is two uniform all-to-alls of
``S / P * H / P * D`` elements per pair.  The reference has no attention or sequence code; this is an example of
the library's collective in the place a training framework would use it.  Both directions are persistent calls:
buffers and counts are fixed at construction, a call is one pack (a strided local copy) and one kernel launch.
When one process hosts every rank there is nobody to pack for: one kernel (``csrc/kernels/reshard.cu``) moves every
element from the caller's tensors to its final place.
"""
from __future__ import annotations

import ctypes as C
from typing import List, Sequence

import numpy as np
import torch

from .. import _native


class UlyssesExchange:
    def __init__(self, comm, seq_local: int, heads: int, head_dim: int, dtype=torch.bfloat16, algo: str = "spreadout",
                 **algo_kw):
        P, L = comm.P, comm.L
        if heads % P:
            raise ValueError("the number of heads must be a multiple of the number of ranks")
        self.comm, self.P, self.L = comm, P, L
        self.s_l, self.h, self.hp, self.d, self.dtype = seq_local, heads, heads // P, head_dim, dtype
        self.block = seq_local * self.hp * head_dim                  # elements per (source, destination) pair
        dev = f"cuda:{comm.device}"
        n = P * self.block
        counts = np.full((L, P), self.block, dtype=np.int32)
        displs = np.tile(np.arange(P, dtype=np.int64) * self.block, (L, 1))
        self._send = [torch.empty(n, dtype=dtype, device=dev) for _ in range(L)]
        self._recv = [comm.symm_empty(n, dtype) for _ in range(L)]
        self._call = comm.prepare(self._send, self._recv, counts, displs, counts, displs, algo=algo, **algo_kw)
        # One process hosting every rank, direct exchange: pack, exchange and unpack are one strided copy, which
        # rbv_reshard_heads does in one launch.  A schedule that the caller asked for, an injected fault or a traced
        # call (other kernels, or none of their stamps) goes through the alltoallv.
        self._direct = (comm.nproc == 1 and P <= 64 and algo == "spreadout" and not algo_kw and self.block > 0
                        and self._call.kind == "static" and not comm.tracing)
        if self._direct:
            self._device = self._recv[0].device
            self._ptrs = C.c_void_p * P
            self._recv_ptrs = self._ptrs(*[t.data_ptr() for t in self._recv])
            starts = [t.data_ptr() for t in self._recv]
            self._recv_span = (min(starts), max(starts) + n * self._recv[0].element_size())
            self._piece_bytes = self.hp * head_dim * self._recv[0].element_size()

    def _as_list(self, x) -> List[torch.Tensor]:
        return [x] if isinstance(x, torch.Tensor) else list(x)

    def _reshard(self, seq_side, head_side, to_head: bool) -> None:
        st = _native.current_stream(self.comm.device)
        rc = self.comm._lib.rbv_reshard_heads(self.comm._ctx, seq_side, head_side, self.s_l, self._piece_bytes,
                                              1 if to_head else 0, st)
        if rc:
            raise RuntimeError(f"re-sharding launch failed (CUDA error {rc})")

    def _plain(self, xs) -> bool:
        """Tensors the kernel can read where they are: packed, of the exchange's type, size and device (anything else
        is converted, broadcast or refused by the copy into the send buffer)."""
        n, dt, dev = self.P * self.block, self.dtype, self._device
        return len(xs) == self.P and all(t.dtype == dt and t.device == dev and t.numel() == n and t.is_contiguous()
                                         and not t.is_conj() and not t.is_neg() for t in xs)

    def seq_to_head(self, x: Sequence[torch.Tensor] | torch.Tensor) -> List[torch.Tensor]:
        """``[S / P, H, D]`` per local rank -> ``[S, H / P, D]`` per local rank (views of the library's buffers,
        valid until the next exchange)."""
        P, s_l, hp, d = self.P, self.s_l, self.hp, self.d
        xs = self._as_list(x)
        if self._direct and self._plain(xs):
            at = [t.data_ptr() for t in xs]
            lo, hi = self._recv_span
            nbytes = P * self.block * xs[0].element_size()
            if all(p + nbytes <= lo or p >= hi for p in at):         # not a view of the result buffers
                self._reshard(self._ptrs(*at), self._recv_ptrs, True)
                return [r.view(P * s_l, hp, d) for r in self._recv]
        for buf, t in zip(self._send, xs):
            # block for rank q = my sequence slice of head group q
            buf.view(P, s_l, hp, d).copy_(t.view(s_l, P, hp, d).permute(1, 0, 2, 3))
        self._call.launch()
        return [r.view(P * s_l, hp, d) for r in self._recv]          # block from rank q = sequence slice q

    def head_to_seq(self, y: Sequence[torch.Tensor] | torch.Tensor) -> List[torch.Tensor]:
        """``[S, H / P, D]`` per local rank -> ``[S / P, H, D]`` per local rank (fresh tensors)."""
        P, s_l, hp, d = self.P, self.s_l, self.hp, self.d
        ys = self._as_list(y)
        if self._direct and self._plain(ys):
            out = [torch.empty((s_l, self.h, d), dtype=self.dtype, device=self._device) for _ in range(P)]
            self._reshard(self._ptrs(*[t.data_ptr() for t in out]), self._ptrs(*[t.data_ptr() for t in ys]), False)
            return out
        for buf, t in zip(self._send, ys):
            buf.copy_(t.reshape(-1))                                 # sequence slice q is already the block for rank q
        self._call.launch()
        # block from rank q = my sequence slice of head group q
        return [r.view(P, s_l, hp, d).permute(1, 0, 2, 3).reshape(s_l, self.h, d) for r in self._recv]
