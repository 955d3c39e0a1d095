"""Shared-exponent groups of auxiliary shells.

The auxiliary shells of one atom and angular momentum usually are contractions of one primitive
set (RICD/acCD sets are: 2 to 6 shells over up to 22 exponents), so every primitive integral
serves all shells of the group.  ``AuxGroups`` collects the shells of a basis (or of a block of
it) by (atom, centre, l, exponent list) and holds the device arrays the group kernels read
(``include/dfb.h``: ``dfb_groups_t``).  A basis without shared exponents gives one group per
shell, for which the kernels do the same work as shell by shell.
"""

from __future__ import annotations

import numpy as np
import torch

from . import _lib

NQ = (1, 4, 16)  # largest primitive counts of a task: one where tasks are few, more where set-up is worth sharing
# first bra entries of the chunk lists (AuxGroups.chunks) by primitive count: integrals take one primitive per task
PLO = {1: ("all", "own", "after"), 4: ("all", "after"), 16: ("all", "after")}


class DevicePool:
    """Host arrays of one type, uploaded together: ``add`` returns a handle, ``upload`` makes the views."""

    def __init__(self, dtype):
        self.dtype = np.dtype(dtype)
        self.parts: list = []
        self.n = 0

    def add(self, a) -> tuple[int, int, tuple]:
        a = np.ascontiguousarray(a, dtype=self.dtype)
        h = (self.n, a.size, a.shape)
        pad = -a.size % 4  # views start on 16-byte boundaries
        self.parts.append(a.ravel())
        if pad:
            self.parts.append(np.zeros(pad, self.dtype))
        self.n += a.size + pad
        return h

    def upload(self, device):
        buf = torch.as_tensor(np.concatenate(self.parts) if self.parts else np.zeros(1, self.dtype), device=device)
        return lambda h: buf[h[0]:h[0] + h[1]].view(h[2])


class AuxGroups:
    def __init__(self, aux, shells, device, cxyz: torch.Tensor, aostart: torch.Tensor, atom: torch.Tensor):
        shells = np.asarray(shells, dtype=np.int64)
        shells = shells[np.argsort(aux.shell_l[shells], kind="stable")]
        groups: dict = {}
        start, count = aux.shell_prim_start, aux.shell_nprim
        for s in shells.tolist():
            a, n = int(start[s]), int(count[s])
            key = (int(aux.shell_l[s]), int(aux.shell_atom[s]), aux.shell_cxyz[s].tobytes(),
                   aux.prim_exp[a:a + n].tobytes())
            groups.setdefault(key, []).append(s)
        info, coef, exps, lists = [], [], [], []
        p0 = c0 = 0
        self.by_l: dict = {}      # l -> group indices (consecutive)
        self.prims: dict = {}     # l -> (first primitive, one past the last)
        for (l, *_), members in groups.items():
            rep = members[0]
            a, n = int(start[rep]), int(count[rep])
            self.by_l.setdefault(l, []).append(len(info))
            info.append((rep, p0, n, len(members), c0, len(lists)))
            exps.append(aux.prim_exp[a:a + n])
            for s in members:
                b = int(start[s])
                coef.append(aux.prim_coef[b:b + n])
            lists += members
            lo, _ = self.prims.get(l, (p0, p0))
            p0 += n
            c0 += n * len(members)
            self.prims[l] = (lo, p0)
        self.info = np.asarray(info, dtype=np.int32).reshape(-1, 6)
        self.nprim = p0
        self.device = device
        cat = lambda v: np.concatenate(v) if v else np.ones(1)  # noqa: E731
        ints, dbls = DevicePool(np.int32), DevicePool(np.float64)
        e = cat(exps)
        z = np.zeros_like(e)
        hd = [dbls.add(a) for a in (cat(coef), e, 1.0 / e,
                                    np.stack([e, 1.0 / e, 2.0 * np.pi ** 2.5 / e, z, z, z, 2.0 * e, z], axis=1))]
        grp = np.repeat(np.arange(len(self.info)), self.info[:, 2])
        hi = [ints.add(a) for a in (self.info, lists or [0], self.info[grp, 0], grp, np.arange(p0), np.ones(p0))]
        hl = {k: ints.add(v) for k, v in self._lists().items()}
        di, dd = ints.upload(device), dbls.upload(device)
        coef_d, exp_d, rexp_d, rec_d = (dd(h) for h in hd)
        info_d, shells_d, rep_d, grp_d, idx_d, one_d = (di(h) for h in hi)
        self._lists_d = {k: di(h) for k, h in hl.items()}
        self._keep = (coef_d, exp_d, rexp_d, rec_d, info_d, shells_d, rep_d, grp_d, idx_d, one_d, cxyz, aostart, atom)
        p = _lib.ptr
        self.c = _lib.Groups(p(info_d), p(coef_d), p(shells_d), p(exp_d), p(rexp_d), p(cxyz), p(aostart), p(atom))
        # the primitives as bra entries of the metric kernels (dfb_bra_t with b_dummy)
        self.bra = _lib.Bra(p(rep_d), p(grp_d), p(idx_d), p(one_d), p(rec_d), p(cxyz), p(aostart), p(atom), 1)
        self.plans: dict = {}  # launch plans of the engine that owns the groups

    def _lists(self) -> dict:
        """Every host list of the groups by key: chunk lists ('c', l, nq, first bra entry), group lists
        ('g', l), group numbers ('i', l), primitive numbers ('p', l)."""
        out = {}
        self._rows = {}
        for l, gs in self.by_l.items():
            inf = self.info[gs].astype(np.int64)
            n, p0 = inf[:, 2], inf[:, 1]
            lo = self.prims[l][0]
            rows = np.concatenate([[0], np.cumsum(n)])
            inf0 = np.asarray(gs)
            out["g", l] = np.stack([inf0, rows[:-1]], axis=1)
            out["i", l] = inf0
            out["p", l] = np.arange(*self.prims[l])
            for nq in NQ:
                cnt = -(-n // nq)  # chunks per group
                first = np.concatenate([[0], np.cumsum(cnt)])
                g = np.repeat(np.arange(len(gs)), cnt)
                k = (np.arange(first[-1]) - first[g]) * nq
                base = np.stack([inf0[g], p0[g] + k, np.minimum(nq, n[g] - k), rows[g] + k, np.zeros_like(k)], axis=1)
                for plo in PLO[nq]:
                    out["c", l, nq, plo] = lst = base if plo == "all" else base.copy()
                    if plo != "all":
                        lst[:, 4] = (p0 - lo if plo == "own" else p0 + n - lo)[g]
                self._rows[l, nq] = (rows, first)
        return out

    def chunks(self, l: int, nq: int, plo: str = "all") -> torch.Tensor:
        """Ranges of at most ``nq`` primitives of the l groups, 5 ints each: group, first primitive, count,
        first row, first bra entry.  Metric with equal l on both sides: the bra primitives used with a group
        start at the group itself (``plo='own'``, integrals) or behind it (``'after'``, derivatives: a group
        with itself has none), so that unordered group pairs occur once."""
        return self._lists_d["c", l, nq, plo]

    def group_rows(self, l: int, nq: int):
        """The l groups: device list of (group, first row), host first rows and first chunks of
        ``chunks(l, nq)`` with the totals at the end."""
        return (self._lists_d["g", l], *self._rows[l, nq])

    def max_shells(self, l: int) -> int:
        return int(self.info[self.by_l[l], 3].max())

    def group_ids(self, l: int) -> torch.Tensor:
        return self._lists_d["i", l]

    def prim_ids(self, l: int) -> torch.Tensor:
        return self._lists_d["p", l]
