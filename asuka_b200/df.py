"""DF integral engine: device-resident bases, pair tables and class task lists.

``DFEngine`` owns everything the Rys kernels of ``libdfb.so`` read for one
(AO basis, aux basis) pair and exposes

* ``metric()``      -> V[P,Q] = (P|Q)                     (naux, naux)
* ``int3c(layout)`` -> X = (mu nu|P) as 'Qmn' (naux,nao,nao) or 'mnQ' (nao,nao,naux)
* ``deriv3c(bar)``  -> sum bar . d(mu nu|P)/dR  accumulated into grad (natm, 3)
* ``deriv2c(bar)``  -> sum bar . d(P|Q)/dR      accumulated into grad (natm, 3)

and the reference's DF-build seams as module functions with the same names and
argument meaning (``asuka/cueri/df.py:803,859,946,994``,
``asuka/integrals/cueri_df.py:33-133``): ``metric_2c2e_basis``,
``int3c2e_basis``, ``cholesky_metric``, ``whiten_3c2e``,
``build_df_B_from_cueri_packed_bases``.

Task enumeration follows the reference's unscreened DF build (every l-ordered
AO shell pair times every aux shell, ``asuka/cueri/gpu.py:1833-1834``; metric
over unordered aux pairs oriented l(P) >= l(Q), ``gpu.py:1590-1706``); the
tasks of one angular class go to the device as a (pairs x aux shells) grid.
"""

from __future__ import annotations

import ctypes
import functools
import os
import weakref

import numpy as np
import torch

from . import _lib
from . import linalg as _la
from .auxgroups import AuxGroups, DevicePool
from .basis import BasisCartSoA, build_shell_pairs_l_order, from_reference_like, ncart

_DATA = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data")
_TABLE_READY: set[int] = set()
PRIM_SCREEN = 1e-20  # primitive-pair magnitude bound below which a pair is skipped (0 = evaluate all)
NSTREAMS = int(os.environ.get("DFB_STREAMS", "8"))  # side streams for per-class launches (2/4/6/8 measured: 8 fastest)
# Doubles of primitive integrals per stream and wave of a class (8 MB; one group up to 32 MB, or over 32 pairs):
# eight streams then stay within L2.  3c integrals at 8 / 64 MB: (H2O)8 4.86 / 4.96 ms, decane 1.88 / 1.86,
# (H2O)3 QZVP 7.85 / 7.77; scratch 71 / 535 MB
PRIM_WAVE = 1 << 20
# Share of dropped elements from which a memset of the tensor is faster than zeros for the dropped blocks, whose rows
# are one AO shell long in 'Qmn' and one aux range in 'mnQ'.  Qmn, blocks / memset: (H2O)8 share 0.18 0.85 / 0.34 ms,
# decane 0.14 0.24 / 0.12, (H2O)3 QZVP 0.06 0.34 / 0.41, (H2O)3 TZVP 0.02 0.015 / 0.025; mnQ: 0.13 / 0.34, 0.04 / 0.12,
# 0.08 / 0.40, 0.014 / 0.024, (H2O)5 share 0.12 0.046 / 0.088 (even at 0.07 and at 0.23 to 0.46)
ZERO_SHARE = (1 / 16, 1 / 4)  # 'Qmn', 'mnQ'
# Lanes of one derivative class from which its tasks take 4 and 16 primitives: a task's set-up (rows, pair data,
# closing sums) is shared, but too few tasks leave SMs idle (2^19 and none: (H2O)8 7.15 ms, decane 2.92;
# 2^17 and 2^20: 6.51 and 2.48)
GRAD_THREADS, GRAD_BIG = 1 << 17, 1 << 20
SEG_PRIMS = 8  # primitive pairs of a derivative task: contracted pairs are cut, so that no task outlasts the rest
NROOTS_SLOTS = 11  # DFB_NROOTS_MAX + 1
_SIDE_STREAMS: dict[int, list] = {}
_SIDE_HANDLES: dict = {}  # device index -> ctypes array of the side streams' handles


class ScratchHolder:
    """Device scratch for the generic shell-by-shell kernels, shared by engines that run one after
    another on the same streams (a batch of molecules): one buffer, grown to the largest need."""

    def __init__(self):
        self.t: torch.Tensor | None = None

    def get(self, need: int, device) -> torch.Tensor:
        if self.t is None or self.t.numel() < need:
            self.t = None
            self.t = torch.empty(need, dtype=torch.float64, device=device)
        return self.t[:need]


@functools.lru_cache(maxsize=1)
def _rys_table_host():
    with np.load(os.path.join(_DATA, "rys_table.npz")) as z:
        nmax, tmax, nint, deg = z["meta"]
        nmax, nint, deg = int(nmax), int(nint), int(deg)
        coefs, herms = [], []
        offs = np.zeros(NROOTS_SLOTS, dtype=np.int32)
        hoffs = np.zeros(NROOTS_SLOTS, dtype=np.int32)
        o = h = 0
        for n in range(1, nmax + 1):
            c = np.ascontiguousarray(z[f"coef{n}"], dtype=np.float64).ravel()
            w = np.ascontiguousarray(z[f"herm{n}"], dtype=np.float64).ravel()
            offs[n], hoffs[n] = o, h
            coefs.append(c)
            herms.append(w)
            o += c.size
            h += w.size
    return np.concatenate(coefs), offs, np.concatenate(herms), hoffs, nmax, nint, deg, float(tmax)


def ensure_rys_table(device: torch.device) -> None:
    """Upload the Rys node/weight table to ``device`` once per process."""
    idx = torch.device(device).index
    idx = torch.cuda.current_device() if idx is None else idx
    if idx in _TABLE_READY:
        return
    coef, offs, herm, hoffs, nmax, nint, deg, tmax = _rys_table_host()
    L = _lib.lib()
    with torch.cuda.device(idx):
        rc = L.dfb_rys_table_init(coef.ctypes.data, offs.ctypes.data, coef.size, herm.ctypes.data, hoffs.ctypes.data,
                                  herm.size, nmax, nint, deg, tmax)
    _lib.check(rc, "dfb_rys_table_init")
    _TABLE_READY.add(idx)


PREC_FP64, PREC_MIXED = 0, 1  # DFB_PREC_FP64 / DFB_PREC_MIXED of include/dfb.h
PREC_ALL_MIXED = -1  # 'mixed_all': every class in FP32 (measurement of the per-class errors)


def _prec_code(precision: str) -> int:
    """'fp64' -> DFB_PREC_FP64; 'mixed' -> DFB_PREC_MIXED for the classes the precision table
    admits (FP64 for the others); 'mixed_all' -> DFB_PREC_MIXED for every class."""
    if precision == "fp64":
        return PREC_FP64
    if precision == "mixed":
        return PREC_MIXED
    if precision == "mixed_all":
        return PREC_ALL_MIXED
    raise ValueError(f"precision must be 'fp64', 'mixed' or 'mixed_all', got {precision!r}")


@functools.lru_cache(maxsize=1)
def mixed_class_table() -> dict:
    """Angular classes whose FP32-component kernels the mixed mode uses, per kind, as sets of
    (la, lb, lc): the 3c integrals ('int3c').  Written by ``asuka_b200.tune_precision`` from the first-order
    energy and gradient errors and the times of every class on the group kernels; classes not listed, the metric
    and the derivative contractions run in FP64 in mixed mode too."""
    p = os.path.join(_DATA, "class_precision.json")
    if not os.path.exists(p):
        return {}
    import json

    with open(p) as f:
        t = json.load(f)
    return {k: {tuple(int(v) for v in c) for c in t.get(k, [])} for k in ("int3c",)}


def _class_prec(code: int, kind: str, la: int, lb: int, lc: int) -> int:
    if code == PREC_FP64:
        return PREC_FP64
    if code == PREC_ALL_MIXED:
        return PREC_MIXED
    return PREC_MIXED if (la, lb, lc) in mixed_class_table().get(kind, ()) else PREC_FP64


def _stream() -> int:
    return _lib.current_stream()


def _as_soa(b) -> BasisCartSoA:
    return b if isinstance(b, BasisCartSoA) else from_reference_like(b)


# dfb_grad_class_t and dfb_prim_class_t, filled as NumPy records
_GRAD_CLASS = np.dtype([(n, "u8" if t is ctypes.c_void_p else "i4") for n, t in _lib.GradClass._fields_], align=True)
_PRIM_CLASS = np.dtype([(n, "u8" if t is ctypes.c_void_p else "i4") for n, t in _lib.PrimClass._fields_], align=True)


@functools.lru_cache(maxsize=4096)
def _group_class(la: int, lb: int, lc: int, metric: bool) -> bool:
    return bool(_lib.lib().dfb_grad_supported(la, lb, lc, int(metric)))


class _PairStatic:
    """What the AO pair lists of every geometry share: the primitive pairs of all shell pairs (owner, index within
    it, and the factors of their magnitude bound), the angular class of each shell pair, and the pairs by
    (class, A, B)."""

    def __init__(self, ao: BasisCartSoA, sp):
        npr = sp.sp_npair.astype(np.int64)
        self.owner = np.repeat(np.arange(sp.nsp), npr)
        self.loc = (np.arange(self.owner.size) - np.repeat(sp.sp_pair_start[:-1].astype(np.int64), npr)).astype(np.int32)
        A, B = sp.sp_A[self.owner], sp.sp_B[self.owner]
        nb = ao.shell_nprim[B]
        pa = ao.shell_prim_start[A] + self.loc // nb
        pb = ao.shell_prim_start[B] + self.loc % nb
        a, b = ao.prim_exp[pa], ao.prim_exp[pb]
        p = a + b
        self.coef = np.abs(ao.prim_coef[pa] * ao.prim_coef[pb])
        self.mexp = -a * b / p
        self.power = (np.pi / p) ** 1.5
        la, lb = ao.shell_l[sp.sp_A].astype(np.int64), ao.shell_l[sp.sp_B].astype(np.int64)
        self.classes, cls = np.unique(la * 16 + lb, return_inverse=True)
        self.cls = cls.astype(np.int64)
        self.order = np.lexsort((sp.sp_B, sp.sp_A, self.cls))


def _stable_order(key: np.ndarray) -> np.ndarray:
    """argsort of an integer key, equal keys in their order (16-bit keys sort by radix)."""
    if key.size and -32768 <= key.min() and key.max() <= 32767:
        key = key.astype(np.int16)
    return np.argsort(key, kind="stable")


def _split_classes(st: _PairStatic, cls: np.ndarray, items: np.ndarray, pool: DevicePool) -> dict:
    """(la, lb) -> pool handle of the items of that class; ``items`` and their classes come ordered by class."""
    out = {}
    cut = np.searchsorted(cls, np.arange(len(st.classes) + 1))
    for i, code in enumerate(st.classes.tolist()):
        if cut[i + 1] > cut[i]:
            out[code // 16, code % 16] = pool.add(items[cut[i]:cut[i + 1]])
    return out


def _with_aux(classes, byl):
    """Class entries with their aux shells: their own, or those of the block (``byl``) where they name none."""
    return [(la, lb, lc, pairs, byl[lc] if auxs is None else auxs) for la, lb, lc, pairs, auxs in classes]


class DFEngine:
    """Device-side state of the DF Rys integrals for one (AO, aux) basis pair."""

    def __init__(self, ao_basis, aux_basis, device=None, atom_coords_bohr: np.ndarray | None = None,
                 prim_screen: float = PRIM_SCREEN, scratch: ScratchHolder | None = None):
        self.device = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        if self.device.type != "cuda":
            raise RuntimeError("DFEngine runs on CUDA devices only (no CPU fallback)")
        ensure_rys_table(self.device)
        ao = _as_soa(ao_basis)
        aux = _as_soa(aux_basis)
        if ao.shell_atom is None or aux.shell_atom is None:
            if atom_coords_bohr is None:
                raise ValueError("bases without shell->atom maps need atom_coords_bohr")
            from .basis import shell_to_atom_map

            ao = from_reference_like(ao, shell_to_atom_map(ao, atom_coords_bohr))
            aux = from_reference_like(aux, shell_to_atom_map(aux, atom_coords_bohr))
        self.ao, self.aux = ao, aux
        self.nao, self.naux = ao.nao, aux.nao
        self.natm = int(max(ao.shell_atom.max(initial=-1), aux.shell_atom.max(initial=-1))) + 1
        self.prim_screen = float(prim_screen)
        if ao.lmax > 8 or aux.lmax > 8:
            raise NotImplementedError("shells with l > 8 are not supported")
        dev = self.device

        # ---- AO side (basis arrays, l-ordered shell pairs) and aux side, one upload per type
        self.sp = build_shell_pairs_l_order(ao)
        ints, dbls = DevicePool(np.int32), DevicePool(np.float64)
        aux_l = aux.shell_l
        ilist = [ao.shell_prim_start, ao.shell_nprim, ao.shell_ao_start, ao.shell_atom, self.sp.sp_A, self.sp.sp_B,
                 aux.shell_prim_start, aux.shell_nprim, aux.shell_ao_start, aux.shell_atom, np.arange(aux.nshell),
                 np.repeat(np.arange(aux.nshell), aux.shell_nprim)]
        by_l = {}
        for l in np.unique(aux_l):
            idx = np.nonzero(aux_l == l)[0]
            by_l[int(l)] = ints.add(idx[np.argsort(-aux.shell_nprim[idx], kind="stable")])
        ih = [ints.add(a) for a in ilist]
        dh = [dbls.add(a) for a in (ao.shell_cxyz, ao.prim_exp, ao.prim_coef, aux.shell_cxyz, aux.prim_exp, aux.prim_coef,
                                    1.0 / np.asarray(aux.prim_exp, dtype=np.float64))]
        di, dd = ints.upload(dev), dbls.upload(dev)
        (self.ao_pstart, self.ao_nprim, self.ao_aostart, self.ao_atom, self.sp_A, self.sp_B, self.ax_pstart,
         self.ax_nprim, self.ax_aostart, self.ax_atom, self.ax_self, self.ax_pp_sp) = (di(h) for h in ih)
        (self.ao_cxyz, self.ao_exp, self.ao_coef, self.ax_cxyz, self.ax_exp, self.ax_coef,
         self.ax_rexp) = (dd(h) for h in dh)
        self.aux_by_l = {l: di(h) for l, h in by_l.items()}
        # (P, dummy) self-pair tables of the shell-by-shell metric kernels
        self.axpt = torch.empty((7, max(int(aux.shell_nprim.sum()), 1)), dtype=torch.float64, device=dev)
        self.ps_aux = _lib.PairSide(
            *[_lib.ptr(t) for t in (self.ax_self, self.ax_self, self.ax_pstart, self.ax_nprim, *self.axpt,
                                    self.ax_cxyz, self.ax_aostart, self.ax_atom)], 1)
        self.axs = _lib.AuxSide(*[_lib.ptr(t) for t in (self.ax_cxyz, self.ax_pstart, self.ax_nprim, self.ax_exp,
                                                        self.ax_coef, self.ax_rexp, self.ax_aostart, self.ax_atom)])
        self._classes2c = None
        self.groups = AuxGroups(aux, np.arange(aux.nshell), dev, self.ax_cxyz, self.ax_aostart, self.ax_atom)
        self._scratch = scratch if scratch is not None else ScratchHolder()
        self._aux_blocks_n = None  # blocks of the aux basis (aux_blocks), which hold for every geometry
        self._pair_static = _PairStatic(ao, self.sp)
        self._build_ao_pairs(ao.shell_cxyz)
        self._build_pair_tables()
        if os.environ.get("DFB_DISABLE_TMPL"):
            self.classes2c  # noqa: B018  (lists of the shell metric kernels, before any capture)

    # ------------------------------------------------------------ class lists
    @property
    def classes2c(self):
        """Metric classes of the shell-by-shell kernels: (lP, lQ, P list, Q list) over the unordered aux shell
        pairs oriented l(P) >= l(Q); built when first asked for (with DFB_DISABLE_TMPL set, by the constructor)."""
        if self._classes2c is None:
            aux_l = self.aux.shell_l
            Pi, Qi = np.tril_indices(self.aux.nshell)
            swap = aux_l[Pi] < aux_l[Qi]
            P, Q = np.where(swap, Qi, Pi), np.where(swap, Pi, Qi)
            lP, lQ = aux_l[P], aux_l[Q]
            self._classes2c = [(int(a), int(c), self._i32(P[sel]), self._i32(Q[sel]))
                               for a in np.unique(lP) for c in np.unique(lQ)
                               if (sel := np.nonzero((lP == a) & (lQ == c))[0]).size]
        return self._classes2c

    # ------------------------------------------------------------ class launches over streams
    def _streams(self):
        """Side streams for class launches: classes write disjoint outputs (or add to the
        gradient atomically), so their kernels may overlap and fill each other's tails."""
        idx = self.device.index if self.device.index is not None else torch.cuda.current_device()
        if idx not in _SIDE_STREAMS:
            _SIDE_STREAMS[idx] = [torch.cuda.Stream(device=self.device) for _ in range(NSTREAMS)]
        return _SIDE_STREAMS[idx]

    def _fork(self):
        """(handle of the current stream, number of side streams, ctypes array of their handles), the side streams
        ordered after the current stream."""
        main = _lib.current_stream(self.device.index)
        if NSTREAMS <= 1:
            return main, 1, (ctypes.c_void_p * 1)(main)
        idx = self.device.index if self.device.index is not None else torch.cuda.current_device()
        arr = _SIDE_HANDLES.get(idx)
        if arr is None:
            arr = _SIDE_HANDLES[idx] = (ctypes.c_void_p * NSTREAMS)(*[int(st.cuda_stream) for st in self._streams()])
        _lib.check(_lib.lib().dfb_fork(main, arr, NSTREAMS), "dfb_fork")
        return main, NSTREAMS, arr

    def _join(self, fork) -> None:
        main, n, arr = fork[:3]
        if NSTREAMS > 1:
            _lib.check(_lib.lib().dfb_join(main, arr, n), "dfb_join")

    @property
    def _i32(self):
        return lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.int32), device=self.device)

    @property
    def _f64(self):
        return lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=self.device)

    def _build_ao_pairs(self, shell_cxyz: np.ndarray) -> None:
        """Primitive-pair lists (screened) and the per-class AO pair lists for a geometry.

        A primitive pair is dropped when |c_a c_b| exp(-ab/(a+b) |AB|^2) (pi/(a+b))^(3/2),
        an upper bound of its overlap-like magnitude, is below ``prim_screen`` (1e-20 by
        default): its contribution to any integral is many orders below the FP64 rounding
        of the integral.  Shell pairs with no primitive pair left are dropped.  The
        reference evaluates every pair (``asuka/cueri/gpu.py:1833-1834``); ``prim_screen=0``
        reproduces that exactly.
        """
        sp, st = self.sp, self._pair_static
        if self.prim_screen > 0.0:
            R2 = ((shell_cxyz[sp.sp_A] - shell_cxyz[sp.sp_B]) ** 2).sum(1)
            bound = st.coef * np.exp(st.mexp * R2[st.owner]) * st.power
            keep = bound >= self.prim_screen
            kept_owner, kept_loc = st.owner[keep], st.loc[keep]
        else:
            kept_owner, kept_loc = st.owner, st.loc
        cnt = np.bincount(kept_owner, minlength=sp.nsp)
        start = np.zeros(sp.nsp, dtype=np.int64)
        np.cumsum(cnt[:-1], out=start[1:])
        live = cnt > 0
        pool = DevicePool(np.int32)
        hs = [pool.add(a) for a in (start, cnt, kept_owner, kept_loc)]
        # pairs of a class by decreasing primitive-pair count: with the aux-major task grid a warp walks pairs of
        # similar cost against one aux shell.  Equal counts by (A, B): neighbouring pairs then read and write
        # neighbouring columns of one 3c row
        order = st.order[live[st.order]]
        top = int(cnt.max(initial=0)) + 1
        order = order[_stable_order(st.cls[order] * top - cnt[order])]
        ph = _split_classes(st, st.cls[order], order, pool)
        # derivative bra entries: segments of at most SEG_PRIMS primitive pairs (their contributions add), by class,
        # decreasing length and (A, B)
        nseg = -(-cnt[st.order] // SEG_PRIMS)
        seg_pair = np.repeat(st.order, nseg)
        k = np.arange(seg_pair.size) - np.repeat(np.cumsum(nseg) - nseg, nseg)
        seg_n = np.minimum(SEG_PRIMS, cnt[seg_pair] - SEG_PRIMS * k)
        gs = [pool.add(a) for a in (sp.sp_A[seg_pair], sp.sp_B[seg_pair], start[seg_pair] + SEG_PRIMS * k, seg_n)]
        seg_cls = st.cls[seg_pair]
        order = _stable_order(seg_cls * (SEG_PRIMS + 1) - seg_n)
        gh = _split_classes(st, seg_cls[order], order, pool)
        ao = self.ao
        size = (ao.shell_l.astype(np.int64) + 1) * (ao.shell_l + 2) // 2
        gone = np.nonzero(~live)[0]
        hz, hn = pool.add(gone), pool.add(size)
        dropped = float((size[sp.sp_A[gone]] * size[sp.sp_B[gone]]).sum()) * 2.0 / max(ao.nao, 1) ** 2
        di = pool.upload(self.device)
        self.sp_pstart, self.sp_npair, self.pp_sp, self.pp_local = (di(h) for h in hs)
        self._dropped = (di(hz), di(hn), dropped)  # pairs without primitives, shell sizes, their share of a 3c row
        self._segs = tuple(di(h) for h in gs)
        self._seg_lists = {key: di(h) for key, h in gh.items()}
        self.n_prim_pairs = int(kept_owner.size)
        self.n_prim_pairs_total = int(st.owner.size)
        self.pt = torch.empty((7, max(self.n_prim_pairs, 1)), dtype=torch.float64, device=self.device)
        self.prec = torch.empty((max(self.n_prim_pairs, 1), 8), dtype=torch.float64, device=self.device)
        p = _lib.ptr
        rest = (p(self.prec), p(self.ao_cxyz), p(self.ao_aostart), p(self.ao_atom), 0)
        self.bra_ao = _lib.Bra(p(self.sp_A), p(self.sp_B), p(self.sp_pstart), p(self.sp_npair), *rest)
        self.bra_seg = _lib.Bra(*[p(t) for t in self._segs], *rest)
        self.ps_ao = _lib.PairSide(
            *[_lib.ptr(t) for t in (self.sp_A, self.sp_B, self.sp_pstart, self.sp_npair, *self.pt, self.ao_cxyz,
                                    self.ao_aostart, self.ao_atom)], 0)
        # dropped shell pairs write nothing: outputs are zero-filled first when any exist
        self.n_dropped_pairs = int(gone.size)
        # (la, lb, lc, AO pair list, aux shell list) per angular class.  A program may assign or edit the list: entries
        # with lists of their own run on the shell kernels (_make_plan)
        self._pairs3c = {key: di(h) for key, h in ph.items()}
        self.classes3c = [(a, b, c, pairs, auxs) for (a, b), pairs in self._pairs3c.items()
                          for c, auxs in self.aux_by_l.items()]

    # ------------------------------------------------------------ helpers
    def _build_pair_tables(self) -> None:
        L = _lib.lib()
        p = _lib.ptr
        npp = self.n_prim_pairs
        rc = L.dfb_pair_tables(p(self.ao_cxyz), p(self.ao_pstart), p(self.ao_nprim), p(self.ao_exp), p(self.ao_coef),
                               p(self.sp_A), p(self.sp_B), p(self.sp_pstart), p(self.pp_sp), p(self.pp_local), npp, 0,
                               *[p(r) for r in self.pt], _stream())
        _lib.check(rc, "dfb_pair_tables(ao)")
        eta, px, py, pz, ck, ea, eb = (p(r) for r in self.pt)
        _lib.check(L.dfb_pair_ext(eta, px, py, pz, ck, ea, eb, npp, p(self.prec), _stream()), "dfb_pair_ext")
        nax = int(self.ax_pp_sp.numel())
        rc = L.dfb_pair_tables(p(self.ax_cxyz), p(self.ax_pstart), p(self.ax_nprim), p(self.ax_exp), p(self.ax_coef),
                               p(self.ax_self), p(self.ax_self), p(self.ax_pstart), p(self.ax_pp_sp), 0, nax, 1,
                               *[p(r) for r in self.axpt], _stream())
        _lib.check(rc, "dfb_pair_tables(aux)")

    def set_coords(self, coords) -> None:
        """Move the shell centres to new atom positions ((natm, 3), bohr).

        Host coordinates (numpy or CPU tensor) also rebuild the screened primitive-pair
        lists for the new geometry; device coordinates update the centres and pair tables
        without a host round trip and keep the lists of the last host geometry (use them
        for small moves, such as finite differences or the timed steps of a fixed
        geometry).
        """
        if isinstance(coords, np.ndarray) or (isinstance(coords, torch.Tensor) and not coords.is_cuda):
            c_np = np.asarray(coords, dtype=np.float64).reshape(-1, 3)
            self._build_ao_pairs(c_np[self.ao.shell_atom])
        coords = torch.as_tensor(coords, dtype=torch.float64).to(device=self.device).reshape(-1, 3)
        self.ao_cxyz.copy_(coords.index_select(0, self.ao_atom.long()))
        self.ax_cxyz.copy_(coords.index_select(0, self.ax_atom.long()))
        self._build_pair_tables()

    def _scratch_for(self, deriv: bool, copies: int = 1) -> torch.Tensor:
        key = (deriv, os.environ.get("DFB_DISABLE_TMPL"), id(self.classes3c))
        cache = self.__dict__.setdefault("_need_cache", {})
        if key in cache:
            return self._scratch.get(cache[key] * copies, self.device)
        L = _lib.lib()
        need = 1
        for la, lb, lc, pairs, auxs in self.classes3c:
            n = L.dfb_rys_scratch_doubles(la, lb, lc, pairs.numel() * auxs.numel(), int(deriv))
            _lib.check(0 if n >= 0 else int(n), "dfb_rys_scratch_doubles")
            need = max(need, n)
        ls, count = np.unique(self.aux.shell_l, return_counts=True)
        for i, lp in enumerate(ls.tolist()):  # unordered aux shell pairs, counted without their lists
            for lq, m in zip(ls[:i + 1].tolist(), count[:i + 1].tolist()):
                pairs = int(count[i]) * m if lq < lp else m * (m + 1) // 2
                n = L.dfb_rys_scratch_doubles(lp, 0, lq, pairs, int(deriv))
                _lib.check(0 if n >= 0 else int(n), "dfb_rys_scratch_doubles")
                need = max(need, n)
        cache[key] = need
        return self._scratch.get(need * copies, self.device)

    def aux_blocks(self, max_naux: int = 256):
        """Contiguous aux-shell blocks of at most ``max_naux`` functions, aligned to shells
        (``asuka/cueri/df.py:2059-2119`` plan_aux_blocks_cart); returns (p0, p1, AuxSide) tuples."""
        if getattr(self, "_aux_blocks_n", None) == max_naux:
            return self._aux_blocks
        aux = self.aux
        nc = [ncart(l) for l in aux.shell_l.tolist()]
        cuts = []  # (first shell, one past the last, functions)
        s0 = 0
        while s0 < aux.nshell:
            s1, tot = s0, 0
            while s1 < aux.nshell and (tot + nc[s1] <= max_naux or s1 == s0):
                tot += nc[s1]
                s1 += 1
            cuts.append((s0, s1, tot))
            s0 = s1
        p0s = [int(aux.shell_ao_start[s0]) for s0, _s1, _t in cuts]
        if len(cuts) == 1 and p0s[0] == 0:  # one block: the engine's own lists
            blocks = [(0, cuts[0][2], (self.axs, self.ax_aostart, self.aux_by_l, self.groups))]
        else:
            pool = DevicePool(np.int32)
            hs, hl = [], []
            for (s0, s1, _t), p0 in zip(cuts, p0s):
                hs.append(pool.add(aux.shell_ao_start - p0))
                l = aux.shell_l[s0:s1]
                hl.append({int(v): pool.add(s0 + np.nonzero(l == v)[0]) for v in np.unique(l)})
            di = pool.upload(self.device)
            shifted = [di(h) for h in hs]
            groups = AuxGroups.blocks(aux, self.groups.shell_ids, [np.arange(s0, s1) for s0, s1, _t in cuts], self.device,
                                      self.ax_cxyz, shifted, self.ax_atom)
            blocks = []
            for (s0, s1, tot), p0, sh, hb, gr in zip(cuts, p0s, shifted, hl, groups):
                axb = _lib.AuxSide(*[_lib.ptr(t) for t in (self.ax_cxyz, self.ax_pstart, self.ax_nprim, self.ax_exp,
                                                           self.ax_coef, self.ax_rexp, sh, self.ax_atom)])
                blocks.append((p0, p0 + tot, (axb, sh, {v: di(h) for v, h in hb.items()}, gr)))
        self._aux_blocks, self._aux_blocks_n = blocks, max_naux
        return blocks

    def int3c_block(self, blk, p0: int, p1: int, out: torch.Tensor | None = None,
                    dropped_zero: bool = False, precision: str = "fp64") -> torch.Tensor:
        """X rows for one aux block as (p1-p0, nao, nao) (streamed DF, ``gpu.py:2742``).

        Entries of screened-out shell pairs are not written; they are zeroed here
        unless ``dropped_zero`` says the buffer already holds zeros there (the set
        of dropped pairs is the same for every block, so a reused buffer needs
        zeroing once).
        """
        axb, _shifted, byl, groups = blk
        nao = self.nao
        X = out if out is not None else torch.empty((p1 - p0, nao, nao), dtype=torch.float64, device=self.device)
        if not dropped_zero:
            self._clear_dropped(X, (nao * nao, nao, 1), p1 - p0)
        self._run_int([self._int3c_work(X, (nao * nao, nao, 1), precision, groups, axb, byl)])
        return X

    def deriv3c_block(self, blk, bar: torch.Tensor, grad: torch.Tensor, precision: str = "fp64") -> torch.Tensor:
        """grad += sum over one aux block of bar[P-p0, mu, nu] d(mu nu|P)/dR (block-local adjoint)."""
        axb, _shifted, byl, groups = blk
        nao = self.nao
        bar = bar.contiguous()
        self._run_deriv([self._deriv3c_work(bar, (nao * nao, nao, 1), grad, precision, groups, axb, byl)], grad)
        return grad

    def _scratch_slices(self, deriv: bool):
        """Scratch for the generic kernels: one slice per side stream (launches overlap)."""
        n = max(NSTREAMS, 1)
        buf = self._scratch_for(deriv, copies=n)
        per = buf.numel() // n
        return [buf[i * per:(i + 1) * per] for i in range(n)]

    def _launch_int(self, la, lb, lc, ps, axs, pairs, auxs, ntask, ngrid, mode, out, strides, prec=PREC_FP64):
        L = _lib.lib()
        # the metric (mode 1) stays FP64: its Cholesky factor whitens everything downstream
        prec = PREC_FP64 if mode == 1 else _class_prec(prec, "int3c", la, lb, lc)
        key = (la, lb, lc, mode, prec)

        def fn(stream, _k=key):
            i = self._slot_of(stream)
            scr = self._slices_int[i]
            rc = L.dfb_rys_int_prec(la, lb, lc, ctypes.byref(ps), ctypes.byref(axs), _lib.ptr(pairs), _lib.ptr(auxs),
                                    ntask, ngrid, mode, prec, _lib.ptr(out), *strides, _lib.ptr(scr), scr.numel(),
                                    stream)
            _lib.check(rc, f"dfb_rys_int {_k}")
        return fn

    def _launch_deriv(self, la, lb, lc, ps, axs, pairs, auxs, ntask, ngrid, mode, bar, strides, grad, prec=PREC_FP64):
        L = _lib.lib()
        prec = _class_prec(prec, "deriv2c" if mode == 1 else "deriv3c", la, lb, lc)
        key = (la, lb, lc, mode, prec)

        def fn(stream, _k=key):
            i = self._slot_of(stream)
            scr = self._slices_der[i]
            rc = L.dfb_rys_deriv_prec(la, lb, lc, ctypes.byref(ps), ctypes.byref(axs), _lib.ptr(pairs),
                                      _lib.ptr(auxs), ntask, ngrid, mode, prec, _lib.ptr(bar), *strides,
                                      _lib.ptr(grad), self.natm, _lib.ptr(scr), scr.numel(), stream)
            _lib.check(rc, f"dfb_rys_deriv {_k}")
        return fn

    def _slot_of(self, stream_ptr: int) -> int:
        if NSTREAMS <= 1:
            return 0
        for i, st in enumerate(self._streams()):
            if int(st.cuda_stream) == stream_ptr:
                return i
        return 0

    # ------------------------------------------------------------ integrals
    def metric(self, out: torch.Tensor | None = None) -> torch.Tensor:
        """V[P, Q] = (P|Q), full symmetric (naux, naux)."""
        naux = self.naux
        V = out if out is not None else torch.empty((naux, naux), dtype=torch.float64, device=self.device)
        self._run_int([self._metric_work(V)])
        # diagonal shell blocks are written from one tile in both orders; make V
        # exactly symmetric as the reference does (cueri_df_cpu.py: V = (V+V^T)/2)
        V.copy_(0.5 * (V + V.T))
        return V

    def int3c(self, layout: str = "Qmn", out: torch.Tensor | None = None, precision: str = "fp64") -> torch.Tensor:
        """X = (mu nu|P): 'Qmn' -> (naux, nao, nao), 'mnQ' -> (nao, nao, naux).

        ``precision='mixed'`` runs the class kernels with FP32 recurrence tables and
        accumulators (``DFB_PREC_MIXED``); the output stays FP64."""
        nao, naux = self.nao, self.naux
        if layout == "Qmn":
            shape, s = (naux, nao, nao), (nao * nao, nao, 1)
        elif layout == "mnQ":
            shape, s = (nao, nao, naux), (1, nao * naux, naux)
        else:
            raise ValueError("layout must be 'Qmn' or 'mnQ'")
        X = out if out is not None else torch.empty(shape, dtype=torch.float64, device=self.device)
        self._clear_dropped(X, s, naux)
        self._run_int([self._int3c_work(X, s, precision)])
        return X

    def deriv3c(self, bar: torch.Tensor, grad: torch.Tensor, layout: str = "Qmn", precision: str = "fp64") -> torch.Tensor:
        """grad += sum_{mu nu P} bar[mu nu P] d(mu nu|P)/dR; bar symmetric in (mu, nu)."""
        nao, naux = self.nao, self.naux
        if layout == "Qmn":
            s = (nao * nao, nao, 1)
        elif layout == "mnQ":
            s = (1, nao * naux, naux)
        else:
            raise ValueError("layout must be 'Qmn' or 'mnQ'")
        bar = bar.contiguous()
        self._run_deriv([self._deriv3c_work(bar, s, grad, precision)], grad)
        return grad

    def deriv2c(self, bar: torch.Tensor, grad: torch.Tensor, precision: str = "fp64") -> torch.Tensor:
        """grad += sum_{P,Q} bar[P,Q] d(P|Q)/dR; bar symmetric."""
        bar = bar.contiguous()
        self._run_deriv([self._deriv2c_work(bar, grad, precision)], grad)
        return grad

    # ------------------------------------------------------------ group-kernel routes
    def _plan(self, kind: str, groups: AuxGroups, precision: str, block: bool = False):
        """Launch plan of one contraction ('int', 'der', or with '2' for the metric) over ``groups``: (ctypes
        class array, its length, the classes left to the shell-by-shell kernels as (la, lb, lc, pairs, auxs),
        scratch), kept with the groups while the class list holds the same entries.

        The group kernels (``dfb_prim_integrals``, ``dfb_grad_contract``) take every class with bra l <= 4
        (the metric: l <= 8).  Left on ``dfb_rys_*_prec``: AO shells above g, 'mixed_all' (which measures the
        FP32 shell kernels) and the generic-kernel switch DFB_DISABLE_TMPL."""
        shells = precision == "mixed_all" or bool(os.environ.get("DFB_DISABLE_TMPL"))
        f32 = frozenset(mixed_class_table().get("int3c", ())) if precision == "mixed" and kind == "int" else None
        key = (kind, shells, f32, block)
        now = () if kind.endswith("2") else self.classes3c
        known = groups.plans.get(key)
        if known is not None:
            ids, plan, _entries = known
            if ids == [*map(id, now)]:  # of entries that the plan keeps alive
                return plan
        if len(groups.plans) > 16:
            groups.plans.clear()
        plan = self._make_plan(kind, groups, shells, f32 or (), block)
        groups.plans[key] = ([*map(id, now)], plan, tuple(now))
        return plan

    def _make_plan(self, kind: str, groups: AuxGroups, shells: bool, f32, block: bool):
        metric, deriv = kind.endswith("2"), kind.startswith("der")
        if metric:
            ls = sorted(groups.fam)
            classes = [(lp, 0, lq, None, None) for lp in ls for lq in ls if lq <= lp]
        elif not block:
            classes = self.classes3c
        else:  # the block's aux shells with the pairs of the class's first entry
            first: dict = {}
            for la, lb, lc, pairs, _auxs in self.classes3c:
                if lc in groups.fam:
                    first.setdefault((la, lb, lc), (la, lb, lc, pairs, None))
            classes = list(first.values())
        new, old = [], []
        for c in classes:
            la, lb, lc, pairs, auxs = c
            # the group kernels evaluate whole classes: all pairs of (la, lb) against all aux shells of lc
            whole = metric or (pairs is self._pairs3c.get((la, lb)) and (auxs is None or auxs is self.aux_by_l.get(lc)))
            (new if whole and not shells and _group_class(la, lb, lc, metric) else old).append(c)
        # the longest single tasks (high bra l, few pairs) first: the numerous low classes fill in behind them
        new.sort(key=lambda c: -(c[0] + c[1]))
        if metric:
            bra = {(l, 0): groups.prim_ids(l) for l in groups.fam}
        else:
            lists = self._seg_lists if deriv else self._pairs3c
            bra = {k: (_lib.ptr(v), int(v.numel())) for k, v in lists.items()}
        recs = []
        for la, lb, lc, _pairs, _auxs in new:
            pairs, n = bra[la, lb]
            same = metric and la == lc
            if deriv:
                lo, hi = groups.prims[lc]
                lanes = n * (hi - lo) * ((la + lb + lc + 1) // 2 + 1)
                nq = 16 if lanes >= GRAD_BIG else 4 if lanes >= GRAD_THREADS else 1
                recs.append((la, lb, lc, n, pairs, *groups.chunk_range(lc, nq, "after" if same else "all"), nq))
            else:
                # one primitive per task: a contracted pair's primitives already make a long one
                chunks, _n = groups.chunk_range(lc, 1, "own" if same else "all")
                lst, rows, first_chunk, ng = groups.group_rows(lc, 1)
                ids, nids = groups.group_ids(la) if metric else (0, 0)
                recs.append((la, lb, lc, n, pairs, chunks, lst, rows, first_chunk, ng, groups.max_shells[lc], ids, nids,
                             groups.prims[la][0] if metric else 0, int((la, lb, lc) in f32)))
        cls, dtype = (_lib.GradClass, _GRAD_CLASS) if deriv else (_lib.PrimClass, _PRIM_CLASS)
        arr = (cls * max(len(new), 1))()
        if recs:
            np.frombuffer(arr, dtype=dtype)[:] = recs
        per = 0 if deriv or not new else int(_lib.lib().dfb_prim_scratch(arr, len(new), PRIM_WAVE))
        return arr, len(new), old, per

    def _int3c_work(self, X, strides, precision, groups=None, axs=None, byl=None):
        block = groups is not None
        groups, axs, byl = groups or self.groups, axs or self.axs, byl or self.aux_by_l
        arr, n, old, per = self._plan("int", groups, precision, block)
        pc = _prec_code(precision)
        rest = [(la, lb, lc, self.ps_ao, axs, pairs, auxs, pairs.numel() * auxs.numel(), -pairs.numel(), 0, X, strides, pc)
                for la, lb, lc, pairs, auxs in _with_aux(old, byl)]
        return self.bra_ao, groups, arr, n, per, X, strides, rest

    def _clear_dropped(self, X, strides, naux) -> None:
        """Zeros where the dropped shell pairs would be: their blocks alone, or the whole tensor where they are
        more than ZERO_SHARE of it."""
        lst, sizes, share = self._dropped
        if not self.n_dropped_pairs:
            return
        if share >= ZERO_SHARE[strides[0] < strides[2]]:
            X.zero_()
            return
        rc = _lib.lib().dfb_zero_pairs(ctypes.byref(self.bra_ao), _lib.ptr(lst), lst.numel(), _lib.ptr(sizes), naux,
                                       _lib.ptr(X), *strides, _stream())
        _lib.check(rc, "dfb_zero_pairs")

    def _metric_work(self, V):
        s = (self.naux, 1, 0)
        arr, n, old, per = self._plan("int2", self.groups, "fp64")
        left = {c[:3] for c in old}
        rest = [(lp, 0, lq, self.ps_aux, self.axs, P, Q, P.numel(), 0, 1, V, s)
                for lp, lq, P, Q in (self.classes2c if old else ()) if (lp, 0, lq) in left]
        return self.groups.bra, self.groups, arr, n, per, V, s, rest

    def _deriv3c_work(self, bar, strides, grad, precision, groups=None, axs=None, byl=None):
        block = groups is not None
        groups, axs, byl = groups or self.groups, axs or self.axs, byl or self.aux_by_l
        arr, n, old, _per = self._plan("der", groups, precision, block)
        pc = _prec_code(precision)
        rest = [(la, lb, lc, self.ps_ao, axs, pairs, auxs, pairs.numel() * auxs.numel(), -pairs.numel(), 0, bar, strides,
                 grad, pc) for la, lb, lc, pairs, auxs in _with_aux(old, byl)]
        return self.bra_seg, groups, arr, n, bar, strides, rest

    def _deriv2c_work(self, bar, grad, precision):
        s = (self.naux, 1, 0)
        arr, n, old, _per = self._plan("der2", self.groups, precision)
        left = {c[:3] for c in old}
        pc = _prec_code(precision)
        rest = [(lp, 0, lq, self.ps_aux, self.axs, P, Q, P.numel(), 0, 1, bar, s, grad, pc)
                for lp, lq, P, Q in (self.classes2c if old else ()) if (lp, 0, lq) in left]
        return self.groups.bra, self.groups, arr, n, bar, s, rest

    def _run_int(self, works, then=None):
        """Run the integral works over the side streams and join.  With a second set ``then`` the current
        stream waits for the first set only; the fork is returned for ``_join`` and holds the scratch until then.

        The rows of primitive integrals belong to the call: they come from the allocator in the order of the
        current stream (of the graph, under capture) and go back to it after the join, so calls from several
        streams or threads and captured calls never share them."""
        L = _lib.lib()
        n = max(NSTREAMS, 1)
        every = works + (then or [])
        if any(w[7] for w in every):
            self._slices_int = self._scratch_slices(False)
        per = (max(w[4] for w in every) + 31) // 32 * 32
        rows = torch.empty(n * per, dtype=torch.float64, device=self.device)
        fork = (*self._fork(), rows)
        streams = fork[2]
        try:
            for batch in (works, then or []):
                for bra, groups, arr, ncls, _per, out, (sP, sM, sN), rest in batch:
                    if ncls:
                        rc = L.dfb_prim_integrals(ctypes.byref(bra), ctypes.byref(groups.c), arr, ncls, _lib.ptr(out), sP,
                                                  sM, sN, _lib.ptr(rows), rows.numel(), streams, n)
                        _lib.check(rc, "dfb_prim_integrals")
                    for i, job in enumerate(rest):
                        self._launch_int(*job)(streams[i % n])
                if batch is works:
                    self._join(fork)
        except BaseException:
            self._join(fork)  # what was launched still writes to its rows
            raise
        return fork

    def _run_deriv(self, works, grad) -> None:
        """Run the derivative works over the side streams and join."""
        L = _lib.lib()
        n = max(NSTREAMS, 1)
        if any(w[6] for w in works):
            self._slices_der = self._scratch_slices(True)
        fork = self._fork()
        streams = fork[2]
        for bra, groups, arr, ncls, bar, (sP, sM, sN), rest in works:
            if ncls:
                rc = L.dfb_grad_contract(ctypes.byref(bra), ctypes.byref(groups.c), arr, ncls, _lib.ptr(bar), sP, sM, sN,
                                         _lib.ptr(grad), self.natm, streams, n)
                _lib.check(rc, "dfb_grad_contract")
            for i, job in enumerate(rest):
                self._launch_deriv(*job)(streams[i % n])
        self._join(fork)

    # ------------------------------------------------------------ overlapped phases of one step
    def metric_cholesky_int3c(self, X: torch.Tensor | None = None, precision: str = "fp64"):
        """V = (P|Q), its Cholesky factor L and X = (mu nu|P) ('Qmn') with the phases overlapped.

        The metric classes go to the side streams first and the 3c classes after them; the
        main stream waits only for the metric launches, symmetrizes V and factorises it while
        the 3c classes still run, then joins.  Same results as metric(), cholesky_metric() and
        int3c() in sequence.
        """
        nao, naux = self.nao, self.naux
        if NSTREAMS <= 1:
            V = self.metric()
            return V, cholesky_metric(V), self.int3c("Qmn", out=X, precision=precision)
        V = torch.empty((naux, naux), dtype=torch.float64, device=self.device)
        X = X if X is not None else torch.empty((naux, nao, nao), dtype=torch.float64, device=self.device)
        self._clear_dropped(X, (nao * nao, nao, 1), naux)
        fork = self._run_int([self._metric_work(V)], [self._int3c_work(X, (nao * nao, nao, 1), precision)])
        try:
            V.copy_(0.5 * (V + V.T))
            L, info = torch.linalg.cholesky_ex(V)
        finally:
            self._join(fork)
        if int(info.item()) != 0:
            raise RuntimeError(f"metric Cholesky failed (leading minor {int(info.item())} not positive definite)")
        return V, L, X

    def deriv3c_2c(self, bar3: torch.Tensor, bar2: torch.Tensor, grad: torch.Tensor,
                   precision: str = "fp64") -> torch.Tensor:
        """deriv3c(bar3 'Qmn') and deriv2c(bar2) as one fan-out (both add into grad atomically)."""
        nao = self.nao
        bar3 = bar3.contiguous()
        bar2 = bar2.contiguous()
        self._run_deriv([self._deriv3c_work(bar3, (nao * nao, nao, 1), grad, precision),
                         self._deriv2c_work(bar2, grad, precision)], grad)
        return grad


# ---------------------------------------------------------------- reference seams

_ENGINES: "weakref.WeakValueDictionary" = weakref.WeakValueDictionary()
_ENGINE_KEEP: dict = {}


def get_engine(ao_basis, aux_basis, device=None) -> DFEngine:
    """Engine cached by (id(ao), id(aux), device) like the reference's plan caches (gpu.py:1602-1612)."""
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    key = (id(ao_basis), id(aux_basis), dev.index)
    eng = _ENGINE_KEEP.get(key)
    if eng is None or eng._bases_ref[0]() is not ao_basis or eng._bases_ref[1]() is not aux_basis:
        eng = DFEngine(ao_basis, aux_basis, device=dev)
        try:
            eng._bases_ref = (weakref.ref(ao_basis), weakref.ref(aux_basis))
        except TypeError:
            eng._bases_ref = (lambda: ao_basis, lambda: aux_basis)
        if len(_ENGINE_KEEP) > 8:
            _ENGINE_KEEP.clear()
        _ENGINE_KEEP[key] = eng
    return eng


def _dummy_ao_for(aux_basis):
    """Metric-only engines still need an AO side; an s shell at the first aux centre works."""
    aux = _as_soa(aux_basis)
    return BasisCartSoA(shell_cxyz=aux.shell_cxyz[:1].copy(), shell_prim_start=np.zeros(1, np.int32),
                        shell_nprim=np.ones(1, np.int32), shell_l=np.zeros(1, np.int32),
                        shell_ao_start=np.zeros(1, np.int32), prim_exp=np.ones(1), prim_coef=np.ones(1),
                        shell_atom=None if aux.shell_atom is None else aux.shell_atom[:1].copy())


def metric_2c2e_basis(aux_basis, *, stream=None, backend: str = "gpu_rys", mode: str = "warp", threads: int = 256,
                      mixed_precision: bool = False, atom_coords_bohr=None) -> torch.Tensor:
    """V[P,Q] = (P|Q) on the current CUDA device (``asuka/cueri/df.py:803``)."""
    if backend not in ("gpu_rys", "gpu_sp", "gpu_ss"):
        raise ValueError("backend must be one of gpu_rys/gpu_sp/gpu_ss")
    aux = _as_soa(aux_basis)
    if aux.shell_atom is None:
        aux = from_reference_like(aux, np.zeros(aux.nshell, np.int32))
    eng = DFEngine(_dummy_ao_for(aux), aux)
    return eng.metric()


def _check_ao_rep(ao_rep: str) -> str:
    if ao_rep not in ("cart", "sph"):
        raise ValueError("ao_rep must be 'cart' or 'sph'")
    return ao_rep


def int3c2e_basis(ao_basis, aux_basis, *, stream=None, backend: str = "gpu_rys", mode: str = "warp",
                  threads: int = 256, mixed_precision: bool = False, layout: str = "mnQ",
                  ao_rep: str = "cart") -> torch.Tensor:
    """X[mu,nu,P] = (mu nu|P) (``asuka/cueri/df.py:859``); layout 'mnQ' or 'Qmn'.

    ``ao_rep='sph'`` returns X over real spherical AOs (the aux index stays Cartesian).
    """
    _check_ao_rep(ao_rep)
    ao, aux = _as_soa(ao_basis), _as_soa(aux_basis)
    if ao.shell_atom is None:
        ao = from_reference_like(ao, np.zeros(ao.nshell, np.int32))
    if aux.shell_atom is None:
        aux = from_reference_like(aux, np.zeros(aux.nshell, np.int32))
    eng = DFEngine(ao, aux)
    if ao_rep == "cart":
        return eng.int3c(layout)
    from .sph import cart2sph_ao_matrix, int3c_cart_to_sph

    return int3c_cart_to_sph(eng.int3c("Qmn"), cart2sph_ao_matrix(ao.shell_l, eng.device),
                             "Qmn").permute(*((1, 2, 0) if layout == "mnQ" else (0, 1, 2))).contiguous()


def cholesky_metric(V: torch.Tensor, *, shift: float = 0.0) -> torch.Tensor:
    """Lower Cholesky factor of the metric.

    The reference's CPU DF build factorises V with no diagonal shift
    (``asuka/integrals/cueri_df_cpu.py:521``); that is the default here, so FP64
    results match the reference CPU path.  A non-zero ``shift`` is added to the
    diagonal first, as the reference's GPU builder does (``cueri_df.py:86-89``).
    """
    Vs = 0.5 * (V + V.T)
    if shift:
        Vs = Vs + float(shift) * torch.eye(V.shape[0], dtype=V.dtype, device=V.device)
    L, info = torch.linalg.cholesky_ex(Vs)
    if int(info.item()) != 0:
        raise RuntimeError(f"metric Cholesky failed (leading minor {int(info.item())} not positive definite)")
    return L


def whiten_3c2e(X: torch.Tensor, L: torch.Tensor, layout: str = "mnQ") -> torch.Tensor:
    """B = X L^-T over the aux index, in place (``asuka/cueri/df.py:994``)."""
    if layout == "mnQ":
        nao = X.shape[0]
        X2 = X.view(nao * nao, -1)
        _la.solve_lower_right_T(L, X2, out=X2)  # B = X L^-T over the last index
        return X
    if layout == "Qmn":
        naux = X.shape[0]
        X2 = X.view(naux, -1)
        _la.solve_lower(L, X2, out=X2)  # B_Q rows = L^-1 X
        return X
    raise ValueError("layout must be 'mnQ' or 'Qmn'")


def build_df_B_from_cueri_packed_bases(ao_basis, aux_basis, *, config=None, layout: str = "mnQ",
                                       ao_rep: str = "cart", profile: dict | None = None, return_L: bool = False):
    """Whitened DF factors B with (mu nu|ls) ~= sum_Q B[mu nu Q] B[ls Q] (``asuka/integrals/cueri_df.py:33``).

    FP64 device tensors; ``layout='mnQ'`` -> (nao, nao, naux), ``'Qmn'`` -> (naux, nao, nao).
    Errors raise RuntimeError/ValueError/NotImplementedError; there is no CPU fallback.
    """
    _check_ao_rep(ao_rep)
    ao, aux = _as_soa(ao_basis), _as_soa(aux_basis)
    if ao.shell_atom is None:
        ao = from_reference_like(ao, np.zeros(ao.nshell, np.int32))
    if aux.shell_atom is None:
        aux = from_reference_like(aux, np.zeros(aux.nshell, np.int32))
    eng = DFEngine(ao, aux)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(5)] if profile is not None else None
    if ev:
        ev[0].record()
    V = eng.metric()
    if ev:
        ev[1].record()
    if ao_rep == "cart":
        X = eng.int3c(layout)
    else:  # real spherical AOs on the AO side; the aux index stays Cartesian
        from .sph import cart2sph_ao_matrix, int3c_cart_to_sph

        X = int3c_cart_to_sph(eng.int3c("Qmn"), cart2sph_ao_matrix(ao.shell_l, eng.device), "Qmn")
        if layout == "mnQ":
            X = X.permute(1, 2, 0).contiguous()
    if ev:
        ev[2].record()
    L = cholesky_metric(V)
    if ev:
        ev[3].record()
    B = whiten_3c2e(X, L, layout)
    if ev:
        ev[4].record()
        torch.cuda.synchronize()
        profile.update(t_metric_s=ev[0].elapsed_time(ev[1]) / 1e3, t_int3c2e_s=ev[1].elapsed_time(ev[2]) / 1e3,
                       t_metric_cholesky_s=ev[2].elapsed_time(ev[3]) / 1e3,
                       t_whiten_s=ev[3].elapsed_time(ev[4]) / 1e3, nao=eng.nao, naux=eng.naux)
    return (B, L) if return_L else B
