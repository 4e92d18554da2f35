"""Key / value cache for generation on packed streams.

Rollouts of the policy-gradient trainers (src/lmms_engine/train in the reference delegates generation to
``transformers``' ``generate`` with its ``DynamicCache``) run here on the packed varlen path: every sequence owns a slab of
``capacity`` rows in one buffer per layer; a forward pass writes the rotated keys and the values of its new tokens behind
the rows already held and attends to the gathered rows of every sequence (``cu_seqlens`` of the keys differ from those
of the queries; the attention kernel aligns its causal mask bottom-right, so new token j of a sequence sees the cached
rows and the new rows up to itself).  A pass that feeds one token per sequence runs all layers in one native call that
reads the slabs in place (``models/decode_path.py``); the gather into the packed layout remains for passes with several
new tokens per sequence on top of cached rows of several sequences.
"""
from __future__ import annotations

from typing import List, Optional, Sequence, Tuple

import torch


class PackedKVCache:
    def __init__(self, n_layers: int, capacities: Sequence[int], device=None):
        self.capacities = [int(c) for c in capacities]
        self.base = [0]
        for c in self.capacities:
            self.base.append(self.base[-1] + c)
        self.lens = [0] * len(self.capacities)
        self.k: List[Optional[torch.Tensor]] = [None] * n_layers
        self.v: List[Optional[torch.Tensor]] = [None] * n_layers
        self.device = device
        self._rows: Optional[Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]] = None
        # layers that carry a recurrent state instead of keys / values (linear attention) keep it here:
        # ``state[layer][sequence]`` is whatever that layer stores (convolution tail, state matrix); a pass replaces an entry
        # and writes into no tensor of it, so a caller may keep one to go back to
        self.state: dict = {}
        self.new_lens: List[int] = []
        self.had: List[int] = []
        self.decode_window = -1
        self._counters: Optional[torch.Tensor] = None

    def advance(self, new_lens: Sequence[int]) -> torch.Tensor:
        """Declare the next forward pass: ``new_lens[i]`` new tokens for sequence ``i`` (0 = none).  Returns the rotary
        positions of the new tokens, packed in sequence order; the pass itself is ``model(..., kv_cache=self)``."""
        new_lens = [int(n) for n in new_lens]
        if len(new_lens) != len(self.lens):
            raise ValueError(f"{len(new_lens)} lengths for a cache of {len(self.lens)} sequences")
        if any(n < 0 for n in new_lens):
            raise RuntimeError(f"new token counts {new_lens}: a pass adds tokens, it takes none away")
        self.new_lens, self.had = new_lens, list(self.lens)
        for i, n in enumerate(new_lens):
            if self.lens[i] + n > self.capacities[i]:
                raise ValueError(f"sequence {i}: {self.lens[i]} cached + {n} new tokens exceed its capacity of {self.capacities[i]}")
            self.lens[i] += n
        if not any(new_lens):
            raise ValueError("a forward pass needs at least one new token")
        self._rows = None
        return self._spread(self.had)

    def _spread(self, starts: Sequence[int]) -> torch.Tensor:
        """``starts[i], starts[i] + 1, ...`` for the new tokens of every sequence, on the cache's device."""
        live = [(s, n) for s, n in zip(starts, self.new_lens) if n]
        if len(live) == 1:
            return torch.arange(live[0][0], live[0][0] + live[0][1], device=self.device)
        # on the host whatever the default device is: pinned memory is host memory
        if max(self.new_lens) == 1:
            host = torch.tensor([s for s, _ in live], device="cpu")
        else:
            host = torch.cat([torch.arange(s, s + n, device="cpu") for s, n in live])
        if self.device is None or torch.device(self.device).type != "cuda":
            return host.to(self.device)
        # from pinned memory: a pageable copy waits for everything queued on the device, once per generated token
        return host.pin_memory().to(self.device, non_blocking=True)

    def _row_tables(self) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]:
        """Rows that this pass' tokens go to, rows that they attend to, and the boundaries of the latter; built once per
        pass, when the first layer asks (the one-call decode path needs none of them)."""
        if self._rows is None:
            # a sequence without new tokens has no query rows, hence no key document either
            live = [i for i, n in enumerate(self.new_lens) if n]
            cu = [0]
            for i in live:
                cu.append(cu[-1] + self.lens[i])
            write = self._spread([b + h for b, h in zip(self.base, self.had)])
            read = write if not any(self.had[i] for i in live) else torch.cat(
                [torch.arange(self.base[i], self.base[i] + self.lens[i]) for i in live]).to(self.device)
            self._rows = (write, read, torch.tensor(cu, dtype=torch.int32, device=self.device), max(self.lens[i] for i in live))
        return self._rows

    def slabs(self, layer: int, n_heads: int, dim: int, dtype: torch.dtype, device) -> Tuple[torch.Tensor, torch.Tensor]:
        """Key and value buffers of a layer, ``[rows of all sequences, n_heads, dim]``; rows past a sequence's length are
        not initialised and never read."""
        if self.k[layer] is None:
            self.k[layer] = torch.empty((self.base[-1], n_heads, dim), dtype=dtype, device=device)
            self.v[layer] = torch.empty_like(self.k[layer])
        return self.k[layer], self.v[layer]

    def decode_counters(self, n: int, device) -> torch.Tensor:
        """Arrival counters of the split-key attention, zero between passes."""
        if self._counters is None or self._counters.numel() < n or self._counters.device != device:
            self._counters = torch.zeros(n, dtype=torch.int32, device=device)
        return self._counters

    def extend(self, layer: int, k: torch.Tensor, v: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, int]:
        """Store this pass' keys / values of ``layer``; returns ``(keys, values, cu_seqlens_k, max_seqlen_k)`` of everything
        the new tokens attend to."""
        if not self.new_lens or k.shape[0] != sum(self.new_lens):
            raise ValueError("call advance() with this pass' token counts before the forward pass")
        write, read, cu_k, max_k = self._row_tables()
        k, v = k.detach(), v.detach()
        if self.k[layer] is None:
            self.k[layer] = k.new_empty((self.base[-1],) + tuple(k.shape[1:]))
            self.v[layer] = v.new_empty((self.base[-1],) + tuple(v.shape[1:]))
        for new, slab in ((k, self.k[layer]), (v, self.v[layer])):  # copying into a slice would cast and broadcast
            if new.dtype != slab.dtype or new.shape[1:] != slab.shape[1:] or new.device != slab.device:
                raise RuntimeError(f"rows of {tuple(new.shape[1:])} {new.dtype} on {new.device} for a cache of {tuple(slab.shape[1:])} "
                                   f"{slab.dtype} on {slab.device}")
        if sum(1 for n in self.new_lens if n) == 1:
            i = next(i for i, n in enumerate(self.new_lens) if n)
            lo, hi = self.base[i] + self.had[i], self.base[i] + self.lens[i]
            self.k[layer][lo:hi].copy_(k)
            self.v[layer][lo:hi].copy_(v)
            if self.had[i]:
                k_all, v_all = self.k[layer][self.base[i]:hi], self.v[layer][self.base[i]:hi]
                if torch.is_grad_enabled():  # the backward pass reads them after a later pass has written into the slab
                    k_all, v_all = k_all.clone(), v_all.clone()
                return k_all, v_all, cu_k, max_k
        else:
            self.k[layer].index_copy_(0, write, k)
            self.v[layer].index_copy_(0, write, v)
        if read is write:  # nothing was cached before this pass: its own rows are all there is
            return k, v, cu_k, max_k
        return self.k[layer].index_select(0, read), self.v[layer].index_select(0, read), cu_k, max_k
