"""The work that a user of this library has it do, as cases that can be timed.

The library builds the Hartree-Fock exchange matrix K of a density P from a screened list of shell
quartets. A program gives the list through the C-ABI's add_* stream in its first self-consistency
step, and from then on either streams it again or replays the recorded list with each new density. A
case is a system (water-like molecules: a cluster, or a periodic cell with its image cells; the l <= 2
or the general-contraction l <= 3 basis), a uniform sample 1/stride of its set quartets, the
precision, and the way the program takes:

  replay       libgint_set_P, libgint_replay, libgint_get_K on a recorded list (each further SCF step)
  open         the same with two spin densities (libgint_set_P_polarized, libgint_get_K_polarized)
  incremental  libgint_set_P(dP), libgint_set_K, libgint_replay_incremental, libgint_get_K
  device       libgint_replay_noalloc on the caller's device buffers and stream
  stream       the whole call stream, item by item: set_P, add_prm .. add_set, get_K
  bulk         the same through libgint_add_set_quartets
  team         the stream of an OpenMP team of callers, one handle each, as CP2K drives the C-ABI
  batch        replay of several independent clusters' quartets held in one handle

The geometry belongs to the case ("system" is its seed) and its screened list is made once per
process: the generator stands in for the calling program. The seed of prepare() draws the
density, which is what changes from one step to the next.
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

from libgint_b200.capi import engine_path, load_engine
from libgint_b200.workload import (CONFIGS, Api, MultiSession, Session, SystemBatch, Workload, driver, set_bulk,
                                   set_fp32_threshold)

_D = ctypes.POINTER(ctypes.c_double)


def _case(name, do, **kw):
    c = dict(do=do, basis=2, n_mol=4, box=12.0, images=1, occ=20, stride=1, system=0, max_prm=16, max_ncontr=4,
             fp32=0.0, tuned=False, threads=1, dp=0.0, systems=1)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _named(config, **kw):
    p = CONFIGS[config]
    return dict(basis=p["basis"], n_mol=p["n_mol"], box=p["box_ang"], images=p["n_img_1d"], occ=p["n_occ"], **kw)


def listed():
    water4, p12, p32 = _named("small_l2"), _named("periodic_l2_small"), _named("periodic_l2")
    p64 = _named("periodic_l3")
    return [
        # one SCF step of a few molecules: launches and latencies are all there is
        _case("replay_water4_l2", "replay", **water4),
        # the same step inside a program that owns its device memory
        _case("device_water4_l2", "device", **water4),
        # the first step of that program: its whole list through the per-item calls
        _case("stream_water4_l2", "stream", **water4),
        # a small periodic cell with the l <= 3 basis in few primitives: every class, few rows in each
        _case("replay_water2_l3", "replay", basis=3, n_mol=2, box=6.5, images=3, occ=16, max_prm=4, max_ncontr=3,
              stride=16),
        # an open-shell step on a dense liquid cell
        _case("open_periodic12_l2", "open", stride=8, **p12),
        # the list of that cell given in bulk calls
        _case("bulk_periodic12_l2", "bulk", stride=16, **p12),
        # one SCF step of a liquid cell, l <= 2
        _case("replay_periodic32_l2", "replay", stride=64, **p32),
        # the headline system: 64 molecules, 125 images, general contractions up to f; FP64
        _case("replay_periodic64_l3", "replay", stride=4096, tuned=True, **p64),
        # and with the small quartets in FP32
        _case("mixed_periodic64_l3", "replay", stride=4096, tuned=True, fp32=1e-5, **p64),
        # a late SCF step of it: the change of K from a small change of P, screened
        _case("incremental_periodic64_l3", "incremental", stride=8192, fp32=1e-5, dp=1e-4, **p64),
        # the list of it streamed by a team of callers
        _case("team_periodic64_l3", "team", stride=65536, fp32=1e-5, threads=4, **p64),
        # many independent clusters of uneven size in one handle
        _case("batch_clusters24", "batch", systems=24, stride=128, occ=5),
    ]


# what draw() takes a system from: (basis, fewest and most molecules, images per direction, periodic)
_RANGES = [(2, 2, 12, 1), (3, 2, 8, 1), (2, 3, 32, 3), (3, 2, 32, 3), (3, 1, 6, 5), (2, 2, 12, 5)]


def draw(rng):
    basis, lo, hi, images = rng.choice(_RANGES)
    m = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    # the liquid's density (a 9.86 A cell for 32 molecules, at least 5 A wide) or the clusters' (12 A for 4)
    box = 12.0 * (m / 4.0) ** (1 / 3) if images == 1 else max(5.0, 9.86 * (m / 32.0) ** (1 / 3))
    sets = m * (11 if basis == 2 else 14)
    want = math.exp(rng.uniform(math.log(5e3), math.log(4e5 if basis == 2 else 1e5)))
    stride = max(1, int(sets ** 4 / 8 * 0.08 * (images ** 2) / 9 / want))
    do = rng.choice(["replay", "replay", "replay", "open", "incremental", "device", "stream", "bulk"])
    max_prm = rng.choice([16, 16, 4, 3])
    return _case(None, do, basis=basis, n_mol=m, box=round(box, 3), images=images, occ=max(1, 4 * m if images > 1 else 5 * m),
                 stride=stride, system=rng.randrange(1, 1 << 30), max_prm=max_prm, max_ncontr=rng.choice([4, 3, 2]),
                 fp32=rng.choice([0.0, 1e-5]) if do in ("replay", "incremental", "stream") else 0.0,
                 dp=10.0 ** rng.uniform(-6, -2) if do == "incremental" else 0.0)


# ---------------------------------------------------------------------------------------
# systems and densities
# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _system_of(basis, n_mol, box, images, occ, stride, system, max_prm, max_ncontr):
    return Workload(None, seed=system, setq_stride=stride, max_prm=max_prm, max_ncontr=max_ncontr, n_mol=n_mol,
                    box_ang=box, periodic=int(images > 1), n_img_1d=images, basis=basis, n_occ=occ)


@functools.lru_cache(maxsize=1)
def _clusters_of(systems, stride, system, occ, max_prm, max_ncontr):
    """Clusters of 2 to 12 molecules, the l <= 2 and l <= 3 bases in turn."""
    rng = random.Random(system)
    wls = []
    for k in range(systems):
        m = rng.randint(2, 12)
        wls.append(Workload(None, seed=1000 * system + k, setq_stride=stride, max_prm=max_prm, max_ncontr=max_ncontr,
                            n_mol=m, box_ang=12.0 * (m / 4.0) ** (1 / 3), periodic=0, n_img_1d=1, basis=3 if k % 2 else 2,
                            n_occ=occ * m))
    return SystemBatch(wls)


def _workloads(case):
    c = case
    if c["do"] == "batch":
        return _clusters_of(c["systems"], c["stride"], c["system"], c["occ"], c["max_prm"], c["max_ncontr"]).wls
    return [_system_of(c["basis"], c["n_mol"], c["box"], c["images"], c["occ"], c["stride"], c["system"], c["max_prm"],
                       c["max_ncontr"])]


def _dense(wl, n_occ, gen, scale=2.0):
    """scale C C^T with C of n_occ orthonormal orbitals."""
    n = wl.n_bf
    C = torch.linalg.qr(torch.randn(n, min(n_occ, n), generator=gen, dtype=torch.float64))[0]
    return (scale * (C @ C.T)).numpy()


def _gen(seed):
    g = torch.Generator()
    g.manual_seed(seed)
    return g


class _State:
    """What a program keeps between calls: its handles, the density and the arrays for K."""

    def __init__(self):
        self.close = []

    def __del__(self):
        for f in self.close:
            f()


def _ptr(a):
    return a.ctypes.data_as(_D)


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()     # replays into device buffers share the library's scratch: one stream


def _check(st):
    if st.lib.libgint_last_error(st.h):
        raise RuntimeError(st.lib.libgint_error_string(st.h).decode())


def _streamed(st):
    """Two builds before the measured ones: the handles' queues (two, in turn) have their size by then."""
    for _ in range(2):
        run(st)
    return st


def prepare(case, seed):
    st = _State()
    st.do, st.fp32 = case["do"], case["fp32"]
    st.lib, api, gen = load_engine(), Api(engine_path()), _gen(seed)
    wls = _workloads(case)
    wl = wls[0]
    P = np.concatenate([w.pack(_dense(w, w.params["n_occ"], gen)) for w in wls])
    st.P, st.n, st.K = P, P.size, np.zeros(P.size)
    if st.do == "team":
        st.session = MultiSession(api, wl, case["threads"], max_mem_mb=1000, team=True)
        st.close.append(st.session.close)
        return _streamed(st)
    if st.do == "batch":
        b = SystemBatch(wls)
        raw = b.setup(api, 40000)
        st.h = ctypes.c_void_p(raw)
        st.close.append(lambda: st.lib.libgint_destroy_handle(ctypes.c_void_p(raw)))
        build = lambda: b.build_K(api, raw)  # noqa: E731
    else:
        st.session = Session(api, wl, max_mem_mb=150 if st.do == "device" else 7000 if st.do in ("stream", "bulk") else 40000)
        st.close.append(st.session.close)
        st.h = ctypes.c_void_p(st.session.h)
        if st.do in ("stream", "bulk"):
            return _streamed(st)
        build = lambda: st.session.build_K(P)  # noqa: E731
    set_fp32_threshold(st.fp32)
    try:
        st.lib.libgint_record(st.h, 1 if st.do == "device" else 2)
        K0 = build()[0]
        st.lib.libgint_record(st.h, 0)
    finally:
        set_fp32_threshold(0.0)
    if case["tuned"]:
        st.lib.libgint_autotune(st.h, None)
    if st.do == "open":
        st.P = wl.pack(_dense(wl, case["occ"] // 2 + 1, gen, 1.0))
        st.Pb, st.Kb = wl.pack(_dense(wl, case["occ"] // 2, gen, 1.0)), np.zeros(st.n)
    elif st.do == "incremental":
        A = torch.randn(wl.n_bf, wl.n_bf, generator=gen, dtype=torch.float64).numpy()
        st.P, st.K0 = case["dp"] * wl.pack(0.5 * (A + A.T)), np.ascontiguousarray(K0)
    elif st.do == "device":
        st.dP, st.dK = torch.from_numpy(P).cuda(), torch.zeros(st.n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    _check(st)
    return st


def run(st):
    lib, do = st.lib, st.do
    if do in ("stream", "bulk", "team"):
        set_fp32_threshold(st.fp32)
        set_bulk(do == "bulk")
        try:
            return st.session.build_K(st.P)[0]
        finally:
            set_fp32_threshold(0.0)
            set_bulk(False)
    if do == "device":
        lib.libgint_replay_noalloc(st.h, st.dP.data_ptr(), st.dK.data_ptr(), st.n, _stream().cuda_stream)
        return st.dK
    if do == "open":
        lib.libgint_set_P_polarized(st.h, _ptr(st.P), _ptr(st.Pb), st.n)
        lib.libgint_replay(st.h)
        lib.libgint_get_K_polarized(st.h, _ptr(st.K), _ptr(st.Kb))
        _check(st)
        return st.K, st.Kb
    lib.libgint_set_P(st.h, _ptr(st.P), st.n)
    if do == "incremental":
        lib.libgint_set_K(st.h, _ptr(st.K0), st.n)
        lib.libgint_replay_incremental(st.h, 1e-11)
    else:
        lib.libgint_replay(st.h)
    lib.libgint_get_K(st.h, _ptr(st.K))
    _check(st)
    return st.K


def work(case):
    """Bytes: the density and K once each way, the list's primitive codes (4), shell (32) and row (24)
    records. Flops: per primitive quartet one G_m, its recursion and image sum, per contraction row the
    contraction, HRR, spherical transform and K update, counted from the recursions."""
    lib, buf = load_engine(), (ctypes.c_double * 8)()
    spins = 2 if case["do"] == "open" else 1
    nbytes = flops = 0.0
    for wl in _workloads(case):
        sq, sets = wl.setq(), wl.sets()
        ls, nls = sets[:, 1][sq[:, :4]], sets[:, 2][sq[:, :4]]
        cls = ls @ np.array([64, 16, 4, 1])
        rows = nls.prod(axis=1).astype(np.float64)
        fl = np.zeros((256, 8))
        for c in np.unique(cls):
            lib.libgint_plan_flops(int(c) >> 6, (int(c) >> 4) & 3, (int(c) >> 2) & 3, int(c) & 3, buf)
            fl[c] = list(buf)
        f, nsh, npr = fl[cls], sq[:, 4], sq[:, 5]
        flops += float(np.sum(npr * (f[:, 0] + f[:, 2] + f[:, 3]) + rows * (npr * f[:, 4] + nsh * f[:, 5] + f[:, 6] + spins * f[:, 7])))
        nbytes += 16.0 * spins * wl.info["flat_size"] + 4.0 * npr.sum() + 32.0 * nsh.sum() + 24.0 * rows.sum()
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------
# the same K in 64 bits from the definition, in plain torch: Hermite Gaussians of every charge
# distribution, the truncated-Coulomb potential's derivatives by quadrature, direct contraction
# ---------------------------------------------------------------------------------------
def _boys(L, T):
    """F_0..F_L(T)."""
    m = L + 0.5
    small = T < 1.0
    Ts, Tl = torch.where(small, T, torch.zeros_like(T)), torch.where(small, torch.ones_like(T), T)
    ser, term = torch.zeros_like(T), torch.ones_like(T)
    for k in range(24):
        ser = ser + term / (2 * L + 2 * k + 1)
        term = term * (-Ts) / (k + 1)
    top = torch.special.gammainc(torch.full_like(Tl, m), Tl) * math.gamma(m) * 0.5 * Tl ** (-m)
    F, e = [torch.where(small, ser, top)], torch.exp(-T)
    for n in range(L - 1, -1, -1):
        F.append((2 * T * F[-1] + e) / (2 * n + 1))
    return torch.stack(F[::-1], 1)


def _truncated(L, T, R):
    """G_0..G_L of the Coulomb operator cut at R (in units of the distributions' width)."""
    G = _boys(L, T)
    x, w = np.polynomial.legendre.leggauss(160)
    x, w = (torch.from_numpy(v).to(T.device) for v in (x, w))
    s = torch.sqrt(T).clamp_min(1e-150)
    lo = ((-9.5 - R) / s).clamp(-1, 1)
    hi = ((9.5 - R) / s).clamp(-1, 1)
    near = torch.nonzero(hi > lo)[:, 0]
    for i in near.split(100000):
        h = 0.5 * (hi[i] - lo[i])[:, None]
        u = 0.5 * (hi[i] + lo[i])[:, None] + h * x
        y = R[i][:, None] + s[i][:, None] * u
        wt = w * h * torch.exp(-y * y)
        a, b, v = torch.ones_like(y), 2 * y, 1 - u * u
        for m in range(L + 1):
            G[i, m] -= (-1) ** m / (2.0 * 4 ** m * math.factorial(m)) * (wt * a).sum(1)
            for k in (2 * m + 1, 2 * m + 2):
                a, b = b, 2 * y * b - 2 * k * a
            wt = wt * v
    return G


def _carts(l):
    return [(l - a, a - z, z) for a in range(l + 1) for z in range(a + 1)]


_SOLID = {0: [[1]], 1: [[0, 1, 0], [0, 0, 1], [1, 0, 0]],
          2: [[0, 1, 0, 0, 0, 0], [0, 0, 0, 0, 1, 0], [-1, 0, 0, -1, 0, 2], [0, 0, 1, 0, 0, 0], [1, 0, 0, -1, 0, 0]],
          3: [[0, 3, 0, 0, 0, 0, -1, 0, 0, 0], [0, 0, 0, 0, 1, 0, 0, 0, 0, 0], [0, -1, 0, 0, 0, 0, -1, 0, 4, 0],
              [0, 0, -3, 0, 0, 0, 0, -3, 0, 2], [-1, 0, 0, -1, 0, 4, 0, 0, 0, 0], [0, 0, 1, 0, 0, 0, 0, -1, 0, 0],
              [1, 0, 0, -3, 0, 0, 0, 0, 0, 0]]}


@functools.lru_cache(maxsize=None)
def _spherical(l):
    """Solid harmonics over the cartesians, each of the norm of a monomial with exponent product one."""
    c, M = _carts(l), np.array(_SOLID[l], dtype=np.float64)
    odd = lambda n: math.prod(range(n, 0, -2)) if n > 0 else 1  # noqa: E731
    S = np.array([[0.0 if any((p + q) % 2 for p, q in zip(a, b)) else math.prod(odd(p + q - 1) for p, q in zip(a, b))
                   for b in c] for a in c])
    return M / np.sqrt(np.einsum("mi,ij,mj->m", M, S, M))[:, None]


@functools.lru_cache(maxsize=None)
def _herm(L):
    """All (t, u, v) of order <= L, and for each but the first: axis, the one below, the one below that, its factor."""
    h = [t for n in range(L + 1) for t in _carts(n)]
    at = {t: i for i, t in enumerate(h)}
    ax, i1, i2, f = [], [], [], []
    for t in h[1:]:
        d = next(q for q in range(3) if t[q])
        one = tuple(v - (q == d) for q, v in enumerate(t))
        two = tuple(v - 2 * (q == d) for q, v in enumerate(t))
        ax.append(d), i1.append(at[one]), i2.append(at.get(two, 0)), f.append(float(t[d] - 1))
    return h, at, ax, i1, i2, f


def _expansion(la, lb, p, PA, PB):
    """[n, spherical pairs, Hermites] of the products of two shells' functions on centres A and B."""
    n = p.shape[0]
    h = _herm(la + lb)[0]
    E = torch.zeros(3, la + 1, lb + 1, la + lb + 2, n, dtype=p.dtype, device=p.device)
    for q in range(3):
        E[q, 0, 0, 0] = 1
        for i in range(la + 1):
            for j in range(lb + 1):
                if i + j == 0:
                    continue
                src, X = (E[q, i - 1, j], PA[:, q]) if i else (E[q, i, j - 1], PB[:, q])
                for t in range(i + j + 1):
                    E[q, i, j, t] = X * src[t] + (t + 1) * src[t + 1] + (src[t - 1] / (2 * p) if t else 0)
    ca, cb = _carts(la), _carts(lb)
    idx = lambda q: ([a[q] for a in ca for b in cb for t in h], [b[q] for a in ca for b in cb for t in h],  # noqa: E731
                     [t[q] for a in ca for b in cb for t in h])
    full = math.prod(E[q][idx(q)] for q in range(3)).reshape(len(ca), len(cb), len(h), n)
    A, B = (torch.from_numpy(_spherical(l)).to(p.device) for l in (la, lb))
    return torch.einsum("ma,kb,abhn->nmkh", A, B, full).reshape(n, -1, len(h))


def _quartets(wl):
    """The list as arrays: set quartets [q, 4], and per primitive quartet its set quartet, images and indices."""
    d = driver()
    d.gd_get_shells.restype = d.gd_get_shell_prims.restype = ctypes.c_long
    L, U = ctypes.POINTER(ctypes.c_long), ctypes.POINTER(ctypes.c_uint32)
    d.gd_get_shells.argtypes = d.gd_get_shell_prims.argtypes = None
    sq = wl.setq()
    img = np.empty((wl.info["n_shells"], 3), dtype=np.int64)
    h = 0
    for q in range(sq.shape[0]):
        h += d.gd_get_shells(ctypes.c_void_p(wl._w), ctypes.c_long(q), img[h:].ctypes.data_as(L))
    code = np.empty(wl.info["n_prims"], dtype=np.uint32)
    at = 0
    for k in range(h):
        at += d.gd_get_shell_prims(ctypes.c_void_p(wl._w), ctypes.c_long(k), code[at:].ctypes.data_as(U))
    shell = np.repeat(np.arange(h), img[:, 2])
    q_of = np.repeat(np.arange(sq.shape[0]), sq[:, 4])[shell]
    prm = np.stack([(code >> s) & 255 for s in (24, 16, 8, 0)], 1).astype(np.int64)
    return sq[:, :4], q_of, img[shell, :2], prm


class _Caller(ctypes.Structure):
    """The generator's table of C-ABI entry points, here Python functions that note what it sets up."""
    _fields_ = [("f", ctypes.c_void_p * 32)]


def _setup_of(wl):
    """What the calling program sets up, from its own set-up calls: range, cell, images and per set (R, Z, l, K)."""
    got, V, I, F = {"sets": []}, ctypes.c_void_p, ctypes.c_int, ctypes.c_double
    num = lambda p, n: np.ctypeslib.as_array(p, (n,)).copy()  # noqa: E731

    def atom(h, i, R, Z, n):
        got["sets"].append([num(R, 3), num(Z, n), 0, None])

    def atom_l(h, i, l, nl, K):
        s = got["sets"][i]
        s[2], s[3] = l, num(K, nl * s[1].size).reshape(nl, -1)

    fns = [ctypes.CFUNCTYPE(V)(lambda: 1), ctypes.CFUNCTYPE(None, V)(lambda h: None),
           ctypes.CFUNCTYPE(None, V, F, _D, I, I)(lambda h, r, c, ld, n: got.update(rc=r)),
           ctypes.CFUNCTYPE(None, V, F)(lambda h, f: None), ctypes.CFUNCTYPE(None, V, I)(lambda h, n: None), None, None,
           ctypes.CFUNCTYPE(None, V, ctypes.c_bool, _D, _D)(lambda h, p, a, b: got.update(h=num(a, 9), hi=num(b, 9))),
           ctypes.CFUNCTYPE(None, V, _D, I)(lambda h, p, n: got.update(img=num(p, 3 * n).reshape(n, 3))),
           ctypes.CFUNCTYPE(None, V, I, _D, _D, I)(atom), ctypes.CFUNCTYPE(None, V, I, I, I, _D)(atom_l)]
    table = _Caller()
    for k, f in enumerate(fns):
        table.f[k + 1] = ctypes.cast(f, V).value if f else None
    driver().gd_setup(wl._w, ctypes.addressof(table), 1)
    for s in got["sets"]:   # every contraction normalised
        Z, l, K = s[1], s[2], s[3]
        S = math.pi ** 1.5 / 2 ** l / (Z[:, None] + Z) ** (1.5 + l)
        s[3] = K / np.sqrt(np.einsum("ca,ab,cb->c", K, S, K))[:, None]
    return got


def _exchange(wl, Ps):
    """K of the packed densities Ps over the workload's list."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    env, (sq, q_of, im, prm) = _setup_of(wl), _quartets(wl)
    sets = env["sets"]
    hm, hi, img, rc = put(env["h"]).reshape(3, 3), put(env["hi"]).reshape(3, 3), put(env["img"]), env["rc"]
    lset, nl = np.array([s[2] for s in sets]), np.array([s[3].shape[0] for s in sets])
    nfn = (2 * lset + 1) * nl
    blk = np.zeros((len(sets), len(sets)), dtype=np.int64)
    blk[np.tril_indices(len(sets))] = np.concatenate([[0], np.cumsum(np.outer(nfn, nfn)[np.tril_indices(len(sets))])[:-1]])
    Rs, Zs, Ks = put(np.stack([s[0] for s in sets])), torch.zeros(len(sets), 16), torch.zeros(len(sets), 4, 16)
    Zs, Ks = Zs.double().to(dev), Ks.double().to(dev)
    for k, s in enumerate(sets):
        Zs[k, :s[1].size], Ks[k, :s[3].shape[0], :s[1].size] = put(s[1]), put(s[3])
    wrap = lambda v: (lambda f: (f - torch.round(f)) @ hm)(v @ hi)  # noqa: E731
    Ps = [put(p) for p in Ps]
    Kout = [torch.zeros_like(p) for p in Ps]

    def place(x, y, ix, iy, l1, l2):
        """Offsets in the packed arrays of the pairs of functions: set x's contraction ix, set y's iy."""
        a = (ix[:, None] * (2 * l1 + 1) + np.arange(2 * l1 + 1))[:, :, None]
        b = (iy[:, None] * (2 * l2 + 1) + np.arange(2 * l2 + 1))[:, None, :]
        low = (x >= y)[:, None, None]
        return np.where(low, blk[x, y][:, None, None] + b * nfn[x][:, None, None] + a,
                        blk[y, x][:, None, None] + a * nfn[y][:, None, None] + b)

    kind = np.concatenate([lset[sq], nl[sq]], 1)
    for kd in np.unique(kind, axis=0):
        ls, ns = [int(v) for v in kd[:4]], [int(v) for v in kd[4:]]
        mine = np.nonzero((kind == kd).all(1))[0]
        L, (l1, l2, l3, l4) = sum(ls), ls
        nrow, nint = int(np.prod(ns)), int(np.prod([2 * l + 1 for l in ls]))
        new = np.full(sq.shape[0], -1)
        new[mine] = np.arange(mine.size)
        sel = np.nonzero(new[q_of] >= 0)[0]
        I = torch.zeros(mine.size, nrow, nint, dtype=torch.float64, device=dev)
        H, at, ax, b1, b2, bf = _herm(L)
        h1, h2 = _herm(l1 + l2)[0], _herm(l3 + l4)[0]
        add = torch.tensor([[at[tuple(p + q for p, q in zip(x, y))] for y in h2] for x in h1], device=dev)
        sign = torch.tensor([(-1.0) ** sum(y) for y in h2], dtype=torch.float64, device=dev)
        bf = torch.tensor(bf, dtype=torch.float64, device=dev)
        width = max(len(h1) * len(h2), nint * len(h2) * 2, len(H) * min(len(img), 8), nrow * nint, 200)
        for ch in np.array_split(sel, max(1, int(sel.size * width / 2.5e7))):
            s4, pr, n12 = sq[q_of[ch]], put(prm[ch]), im[ch]
            A, B0, C, D0 = (Rs[put(s4[:, k])] for k in range(4))
            za, zb, zc, zd = (Zs[put(s4[:, k]), pr[:, k]] for k in range(4))
            B, D = A + wrap(B0 - A) + img[put(n12[:, 0])], C + wrap(D0 - C) + img[put(n12[:, 1])]
            p, q = za + zb, zc + zd
            P, Q = (za[:, None] * A + zb[:, None] * B) / p[:, None], (zc[:, None] * C + zd[:, None] * D) / q[:, None]
            rho = p * q / (p + q)
            pre = 2 * math.pi ** 2.5 / (p * q * torch.sqrt(p + q)) * torch.exp(
                -za * zb / p * ((A - B) ** 2).sum(1) - zc * zd / q * ((C - D) ** 2).sum(1))
            X = wrap(P - Q)[:, None, :] - img[None]
            T, R = rho[:, None] * (X * X).sum(2), rc * torch.sqrt(rho)[:, None]
            near = torch.nonzero(T <= R * R + 11 * R + 50)
            Rsum = torch.zeros(ch.size, len(H), dtype=torch.float64, device=dev)
            rest = torch.zeros(ch.size, 1, dtype=torch.float64, device=dev)
            for nr in near.split(max(1, int(2e7 / len(H)))):
                i, x = nr[:, 0], X[nr[:, 0], nr[:, 1]]
                G = _truncated(L, T[nr[:, 0], nr[:, 1]], R[i, 0]) * pre[i, None]
                keep = G[:, :1] > 1e-12     # an image below counts in (00|00) only
                rest.index_add_(0, i, G[:, :1] * ~keep)
                G = G * keep * (-2 * rho[i, None]) ** torch.arange(L + 1, device=dev)
                r = G[:, L:L + 1]
                for m in range(L - 1, -1, -1):
                    k = len(_herm(L - m)[0]) - 1
                    lower = torch.cat([r, r.new_zeros(r.shape[0], k + 1 - r.shape[1])], 1)
                    r = torch.cat([G[:, m:m + 1], x[:, ax[:k]] * lower[:, b1[:k]] + bf[:k] * lower[:, b2[:k]]], 1)
                Rsum.index_add_(0, i, r)
            U = _expansion(l1, l2, p, P - A, P - B) @ (Rsum[:, add] * sign)
            V = U @ _expansion(l3, l4, q, Q - C, Q - D).transpose(1, 2)
            if l1 == 0 and l3 == 0:
                mono = lambda v, l: torch.stack([(v ** put(np.array(c, float))).prod(1) for c in _carts(l)], 1) @ put(_spherical(l)).T  # noqa: E731
                V = V + (rest * mono(A - B, l2))[:, :, None] * mono(C - D, l4)[:, None, :]
            co = [Ks[put(s4[:, k])[:, None], torch.arange(ns[k], device=dev), pr[:, k:k + 1]] for k in range(4)]
            W = torch.einsum("na,nb,nc,nd->nabcd", *co).reshape(ch.size, nrow, 1)
            I.index_add_(0, put(new[q_of[ch]]), W * V.reshape(ch.size, 1, nint))
        i, j, k, l = (np.repeat(sq[mine, c], nrow) for c in range(4))
        ia, ib, ic, id_ = (np.tile(v, mine.size) for v in np.unravel_index(np.arange(nrow), ns))
        fac = 2.0 * np.where(i == j, 0.5, 1) * np.where(k == l, 0.5, 1) * np.where((i == k) & (j == l), 0.5, 1)
        V = -put(fac)[:, None, None, None, None] * I.reshape(-1, 2 * l1 + 1, 2 * l2 + 1, 2 * l3 + 1, 2 * l4 + 1)
        pac, pad = put(place(i, k, ia, ic, l1, l3)), put(place(i, l, ia, id_, l1, l4))
        pbc, pbd = put(place(j, k, ib, ic, l2, l3)), put(place(j, l, ib, id_, l2, l4))
        for Pm, Km in zip(Ps, Kout):
            for src, dst, how in ((pac, pbd, "nac,nabcd->nbd"), (pad, pbc, "nad,nabcd->nbc"), (pbc, pad, "nbc,nabcd->nad"),
                                  (pbd, pac, "nbd,nabcd->nac")):
                Km.index_add_(0, dst.reshape(-1), torch.einsum(how, Pm[src], V).reshape(-1))
    return [K.cpu().numpy() for K in Kout]


def exact(case, seed):
    wl = _workloads(case)[0]
    if case["do"] in ("batch", "team", "incremental") or wl.info["n_shells"] > 100_000 or wl.info["n_prims"] * wl.info["Ng"] > 8_000_000:
        return None
    gen = _gen(seed)
    P = wl.pack(_dense(wl, wl.params["n_occ"], gen))
    if case["do"] == "open":
        return tuple(_exchange(wl, [wl.pack(_dense(wl, case["occ"] // 2 + 1, gen, 1.0)), wl.pack(_dense(wl, case["occ"] // 2, gen, 1.0))]))
    return _exchange(wl, [P])[0]
