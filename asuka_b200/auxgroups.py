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


def shell_group_ids(aux) -> np.ndarray:
    """Per shell: the number of its group, shells with one (l, atom, centre, exponent list) having the same."""
    ids: dict = {}
    start, end = aux.shell_prim_start.tolist(), (aux.shell_prim_start + aux.shell_nprim).tolist()
    keys = zip(aux.shell_l.tolist(), aux.shell_atom.tolist(), map(bytes, np.ascontiguousarray(aux.shell_cxyz)),
               start, end)
    exps = np.ascontiguousarray(aux.prim_exp, dtype=np.float64)
    return np.array([ids.setdefault((l, at, c, exps[a:b].tobytes()), len(ids)) for l, at, c, a, b in keys],
                    dtype=np.int64)


def _ranges(start: np.ndarray, count: np.ndarray) -> np.ndarray:
    """start[0], start[0] + 1, ... (count[0] values), start[1], ..."""
    return np.arange(count.sum()) + np.repeat(start - (np.cumsum(count) - count), count)


class AuxGroups:
    """The groups of one set of shells.  ``blocks`` makes those of several sets at once: one upload, one numbering
    of groups and primitives, and lists that are ranges of common ones."""

    def __init__(self, aux, shells, device, cxyz: torch.Tensor, aostart: torch.Tensor, atom: torch.Tensor):
        _build([self], aux, shell_group_ids(aux), [shells], device, cxyz, [aostart], atom)

    @classmethod
    def blocks(cls, aux, ids: np.ndarray, shells, device, cxyz: torch.Tensor, aostarts, atom: torch.Tensor) -> list:
        """One object per entry of ``shells``, with its own first functions of the shells (``aostarts``); ``ids`` as
        ``shell_group_ids`` gives them (``shell_ids`` of an object over the whole basis)."""
        out = [cls.__new__(cls) for _ in shells]
        _build(out, aux, ids, shells, device, cxyz, aostarts, atom)
        return out

    def chunk_range(self, l: int, nq: int, plo: str = "all") -> tuple[int, int]:
        """Address and length of a list of ranges of at most ``nq`` primitives of the l groups, 5 ints each: group,
        first primitive, count, first row, first bra entry.  Metric with equal l on both sides: the bra primitives
        used with a group start at the group itself (``plo='own'``, integrals) or behind it (``'after'``,
        derivatives: a group with itself has none), so that unordered group pairs occur once."""
        base, first = self._chunks[nq, plo], self._first[nq]
        f, g0, g1 = self.fam[l]
        lo, hi = first[1][f], first[1][f] + first[0][g1 + f]
        return base + 20 * int(lo), int(hi - lo)

    def group_rows(self, l: int, nq: int) -> tuple[int, int, int, int]:
        """The l groups: address of (group, first row) on the device, host addresses of the first rows and of the
        first chunks of ``chunk_range(l, nq)`` with the totals at the end, and the number of groups."""
        f, g0, g1 = self.fam[l]
        at = 8 * (g0 + f)
        return (self._glist + 8 * g0, self._rows.ctypes.data + at, self._first[nq][0].ctypes.data + at, g1 - g0)

    def group_ids(self, l: int) -> tuple[int, int]:
        """Device address and length of the numbers of the l groups."""
        _f, g0, g1 = self.fam[l]
        return self._index + 4 * g0, g1 - g0

    def prim_ids(self, l: int) -> tuple[int, int]:
        """Device address and length of the numbers of the l groups' primitives."""
        lo, hi = self.prims[l]
        return self._index + 4 * lo, hi - lo


def _build(objs, aux, ids, shells, device, cxyz, aostarts, atom) -> None:
    shells = [np.asarray(s, dtype=np.int64) for s in shells]
    S = np.concatenate(shells)
    blk = np.repeat(np.arange(len(shells)), [len(s) for s in shells])
    order = np.lexsort((aux.shell_l[S], blk))  # by block and l, equal ones in their order
    S, blk = S[order], blk[order]
    nprim, start = aux.shell_nprim.astype(np.int64), aux.shell_prim_start.astype(np.int64)
    # groups in the order of their first shells
    _u, first, inv = np.unique(blk * (int(ids.max(initial=0)) + 1) + ids[S], return_index=True, return_inverse=True)
    number = np.empty(len(first), dtype=np.int64)
    number[np.argsort(first)] = np.arange(len(first))
    g = number[inv]
    first = np.sort(first)
    ng = len(first)
    rep, gblk = S[first], blk[first]
    gl = aux.shell_l[rep].astype(np.int64)
    n, ns = nprim[rep], np.bincount(g, minlength=ng)
    members = S[np.argsort(g, kind="stable")]
    p0, c0, s0 = (np.cumsum(v) - v for v in (n, n * ns, ns))
    info = np.stack([rep, p0, n, ns, c0, s0], axis=1)
    # families: the groups of one block and l, consecutive
    new = np.ones(ng, dtype=bool)
    new[1:] = (gblk[1:] != gblk[:-1]) | (gl[1:] != gl[:-1])
    f0 = np.nonzero(new)[0]
    fam = np.cumsum(new) - 1
    f1 = np.append(f0[1:], ng)
    row = p0 - p0[f0][fam] if ng else p0  # rows of a family: its primitives
    at = np.arange(ng) + fam              # per-family lists with a total at the end

    def totals(v, end):
        out = np.zeros(ng + len(f0), dtype=np.int64)
        out[at], out[f1 + np.arange(len(f0))] = v, end
        return out

    ptot = int(n.sum())
    hi = np.append(p0, ptot)[f1] if ng else f1
    rows = totals(row, hi - p0[f0] if ng else hi)
    e = aux.prim_exp[_ranges(start[rep], n)] if ng else np.ones(1)
    coef = aux.prim_coef[_ranges(start[members], nprim[members])] if ng else np.ones(1)
    z = np.zeros_like(e)
    grp = np.repeat(np.arange(ng), n)
    ints, dbls = DevicePool(np.int32), DevicePool(np.float64)
    hd = [dbls.add(a) for a in (coef, e, 1.0 / e,
                                np.stack([e, 1.0 / e, 2.0 * np.pi ** 2.5 / e, z, z, z, 2.0 * e, z], axis=1))]
    hi_ = [ints.add(a) for a in (info, members, rep[grp], np.arange(max(ng, ptot, 1)), grp, np.ones(max(ptot, 1)),
                                 np.stack([np.arange(ng), row], axis=1))]
    hc, firsts = {}, {}
    for nq in NQ:
        cnt = -(-n // nq)  # chunks per group
        c_first = np.cumsum(cnt) - cnt
        of = np.repeat(np.arange(ng), cnt)
        k = (np.arange(of.size) - c_first[of]) * nq
        base = np.stack([of, p0[of] + k, np.minimum(nq, n[of] - k), row[of] + k, np.zeros_like(k)], axis=1)
        for plo in PLO[nq]:
            hc[nq, plo] = lst = base if plo == "all" else base.copy()
            if plo != "all":
                lst[:, 4] = (row if plo == "own" else row + n)[of]
            hc[nq, plo] = ints.add(lst)
        end = np.append(c_first, of.size)
        lo = c_first[f0] if ng else f0
        firsts[nq] = (totals(c_first - lo[fam] if ng else c_first, end[f1] - lo), lo)
    di, dd = ints.upload(device), dbls.upload(device)
    p = _lib.ptr
    coef_d, exp_d, rexp_d, rec_d = (dd(h) for h in hd)
    info_d, members_d, rep_d, index_d, grp_d, one_d, glist_d = (di(h) for h in hi_)
    chunks = {key: p(di(h)) for key, h in hc.items()}
    most = np.maximum.reduceat(ns, f0) if ng else ns
    keep = (coef_d, rep_d, cxyz, atom)
    for b, (o, aostart) in enumerate(zip(objs, aostarts)):
        o.shell_ids = ids
        o.device = device
        o.fam = {}          # l -> (family, first group, one past the last)
        o.prims = {}        # l -> (first primitive, one past the last)
        o.max_shells = {}   # l -> largest shell count of a group
        for f in np.nonzero(gblk[f0] == b)[0].tolist():
            l = int(gl[f0[f]])
            o.fam[l] = (f, int(f0[f]), int(f1[f]))
            o.prims[l] = (int(p0[f0[f]]), int(hi[f]))
            o.max_shells[l] = int(most[f])
        o._chunks, o._first, o._rows = chunks, firsts, rows
        o._glist, o._index = p(glist_d), p(index_d)
        o._keep = (*keep, aostart)  # the pools' buffers live on through their views
        o.c = _lib.Groups(p(info_d), p(coef_d), p(members_d), p(exp_d), p(rexp_d), p(cxyz), p(aostart), p(atom))
        # the primitives as bra entries of the metric kernels (dfb_bra_t with b_dummy)
        o.bra = _lib.Bra(p(rep_d), p(grp_d), p(index_d), p(one_d), p(rec_d), p(cxyz), p(aostart), p(atom), 1)
        o.plans = {}  # launch plans of the engine that owns the groups
