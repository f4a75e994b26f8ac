"""The device memory behind the cache manager: for each group one array
`[layers, 1 + pages + 1, 2 (k, v), kv_heads, page_size, head_dim]` (a layer's slice
without its first and last page is what its kernels get; inside a page the layout is
head-major, so the keys of one (page, head) are one dense `[page_size, head_dim]` tile;
the two pages around a layer's own are guard bands: they hold a fixed pattern that no
kernel may touch, `check_guards` looks at them), and for each layer with a
fixed-size state one array `[slots + 1, *shape]` (the last row is nobody's); and the
slots' own rows: last token, sampler record, recent tokens (the reference keeps these on
the host, bin/reinfer/src/sched_loop.rs:464-485, and only transient `[B]` rows on the
device, crates/cuda/src/engine.rs:1854-1875).
(The reference keeps one f16 buffer, K region then V region, layer folded into the
page index: crates/cuda/src/decode.rs:664-698.)
"""
from __future__ import annotations

from typing import Dict, List, Sequence

import torch

from .. import ops
from .manager import CacheManager


SLOT_RECORD_BYTES = 64          # sizeof(RbSampleParams); the sampler checks it against the library
SLOT_HISTORY = 64               # tokens of the penalty window a slot can hold
GUARD_PATTERN = 0x5A5A          # every 16 bits of a guard page


class CacheStorage:
    def __init__(self, manager: CacheManager, dtype: torch.dtype, device):
        self.manager = manager
        self.dtype = dtype
        self.device = torch.device(device)
        self.group_arrays: List[torch.Tensor] = []
        self.layer_kv: Dict[str, torch.Tensor] = {}
        for g in manager.groups:
            if g.spec.value_dim == g.spec.head_dim:
                page_shape = (2, g.spec.kv_heads, manager.page_size, g.spec.head_dim)
            else:                                   # keys [kv_heads, page, d], then values [kv_heads, page, dv]
                page_shape = (g.spec.page_elems(manager.page_size),)
            arr = torch.zeros((len(g.layers), g.pool.total + 2) + page_shape, dtype=dtype, device=self.device)
            for edge in (0, g.pool.total + 1):
                arr[:, edge].view(torch.int16).fill_(GUARD_PATTERN)
            self.group_arrays.append(arr)
            for li, name in enumerate(g.layers):
                self.layer_kv[name] = arr[li, 1:g.pool.total + 1]          # page -1 and page `total` are the guards
        # a layer's state: one tensor, or (for a mixer that keeps several) a dict of them, nested as its spec is
        self.layer_state: Dict[str, object] = {}

        def make(spec):
            if isinstance(spec, dict):
                return {k: make(v) for k, v in spec.items()}
            sdt = dtype if spec.dtype == "act" else getattr(torch, spec.dtype)
            # one row more than there are slots: the last row belongs to nobody (padding rows of a captured
            # decode step point at it, so that they disturb no request's state)
            return torch.zeros((manager.max_seqs + 1,) + tuple(spec.shape), dtype=sdt, device=self.device)

        for name, spec in manager.states.items():
            self.layer_state[name] = make(spec)
        self.inert_slot = manager.max_seqs
        tensors = self.state_tensors()
        # where the rows of these tensors lie, for the kernel that sets a request's to zero
        self._zero_rows = ops.zero_slots_table(tensors, self.device) if tensors else None
        # the request slots' own rows (as many, plus nobody's): the token last drawn for the request, the sampler's
        # record (parameters, seed, count of draws: csrc/sampler.cu RbSampleParams) and its ring of recent tokens.
        # The sampler kernel reads and writes them; the host writes a row when a request is admitted.
        self.slot_token = torch.zeros(manager.max_seqs + 1, dtype=torch.int32, device=self.device)
        self.slot_records = torch.zeros((manager.max_seqs + 1, SLOT_RECORD_BYTES), dtype=torch.uint8, device=self.device)
        self.slot_history = torch.zeros((manager.max_seqs + 1, SLOT_HISTORY), dtype=torch.int32, device=self.device)

    def check_guards(self) -> List[str]:
        """The guard pages that no longer hold their pattern, as "layer name: before|after" (empty: all intact).
        A page index of -1 or of the pool's size that reached a store would show here.  Synchronises; for tests
        and for looking into a fault, not for every step."""
        bad = []
        for g, arr in zip(self.manager.groups, self.group_arrays):
            for which, edge in (("before", 0), ("after", g.pool.total + 1)):
                touched = (arr[:, edge].reshape(len(g.layers), -1).view(torch.int16) != GUARD_PATTERN).any(dim=1).tolist()
                bad += [f"{name}: {which}" for name, t in zip(g.layers, touched) if t]
        return bad

    def zero_slots(self, slots: Sequence[int]) -> None:
        """A fixed-size state starts at zero when its request is admitted."""
        if self._zero_rows is not None and slots:
            ops.zero_slots(*self._zero_rows, slots)

    def state_tensors(self) -> List[torch.Tensor]:
        out: List[torch.Tensor] = []

        def walk(x):
            if isinstance(x, dict):
                for v in x.values():
                    walk(v)
            else:
                out.append(x)

        for s in self.layer_state.values():
            walk(s)
        return out

    def bytes(self) -> int:
        return sum(a.numel() * a.element_size() for a in self.group_arrays) + \
            sum(a.numel() * a.element_size() for a in self.state_tensors())

    @staticmethod
    def bytes_per_page(manager_groups, page_size: int, dtype: torch.dtype) -> int:
        isz = torch.empty((), dtype=dtype).element_size()
        return sum(len(g.layers) * g.spec.page_elems(page_size) * isz for g in manager_groups)
