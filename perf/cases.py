"""What the speed of this framework is measured on.

The cases are the calls a user of the framework makes, through the Python
layer, from the smallest sector of the tests to the headline sector of the
benchmark:

  apply     y = H x on device vectors (complex128, complex64, and native Q64
            mantissas), reference or tensor order, plain or affine
            (y = scale (H - shift) x + beta z);
  host      the same on page-locked host vectors (mb_op_apply_host), the call
            a reference driver on the CPU makes;
  ground    find_min_eigenpair: plain Lanczos with its Ritz vector, or complex64
            vectors with the FP64 refinement of the energy;
  evolve    time_evolve_state: Krylov exp(-i t H) psi;
  moments   kpm_dos_moments: Chebyshev moments of the density of states;
  momentum  y = H x in a total-momentum sector;
  batch     batch_ground_states: many small sectors on one kept engine.

`exact` restates each in 64 bits with torch alone: states enumerated and sorted
here, H applied hop by hop.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import manybody_gb300 as mb

PREC = {"f64": mb.PREC_F64, "f32": mb.PREC_F32, "q64": mb.PREC_Q64}
ORDER = {"reference": mb.ORDER_REFERENCE, "tensor": mb.ORDER_TENSOR}


def listed():
    return [
        # the smoke test's sector (4,900 states): latency of one call, as in a
        # loop of a user's own driver over small systems
        dict(name="apply_f64_1d8_4+4", kind="apply", lattice="8", n_up=4, n_down=4, u=4.0,
             prec="f64", order="reference", affine=False),
        # an odd filling of a served lattice (792 x 495 states), one step of a
        # user's own three-term recurrence in the engine's order
        dict(name="affine_f64_3x4_5+4", kind="apply", lattice="3x4", n_up=5, n_down=4, u=8.0,
             prec="f64", order="tensor", affine=True),
        # the benchmark's sector (64,128,064 states) by the default call
        dict(name="apply_f64_4x4_6+6", kind="apply", lattice="4x4", n_up=6, n_down=6, u=8.0,
             prec="f64", order="reference", affine=False),
        # complex64 vectors on a ring (11,778,624 states)
        dict(name="apply_f32_1d14_7+7", kind="apply", lattice="14", n_up=7, n_down=7, u=4.0,
             prec="f32", order="reference", affine=False),
        # the benchmark's headline: native Q64 mantissas, 4x4 6+6
        dict(name="apply_q64_4x4_6+6", kind="apply", lattice="4x4", n_up=6, n_down=6, u=8.0,
             prec="q64", order="tensor", affine=False),
        # a CPU driver's call: complex128 host vectors (19,079,424 states)
        dict(name="host_f64_4x4_5+5", kind="host", lattice="4x4", n_up=5, n_down=5, u=8.0,
             prec="f64"),
        # ground state and its vector of a batch-sized sector (63,504 states)
        dict(name="ground_f64_1d10_5+5", kind="ground", lattice="10", n_up=5, n_down=5, u=4.0,
             prec="f64", steps=50, refine=False),
        # the precision path on a large sector: complex64 Lanczos vectors, their Ritz
        # vector, FP64 refinement of its energy
        dict(name="ground_f32_4x4_5+5", kind="ground", lattice="4x4", n_up=5, n_down=5, u=8.0,
             prec="f32", steps=40, refine=True),
        # a time step of a mid-size sector (853,776 states)
        dict(name="evolve_f64_3x4_6+6", kind="evolve", lattice="3x4", n_up=6, n_down=6, u=4.0,
             prec="f64", time=0.4, order="reference"),
        # density of states, one probe (3,312,400 states)
        dict(name="moments_q64_4x4_4+4", kind="moments", lattice="4x4", n_up=4, n_down=4, u=8.0,
             prec="q64", moments=128),
        # total momentum (0,0) of 4x4 5+5 (1,192,464 states, about 200 entries a row)
        dict(name="momentum_f64_4x4_5+5", kind="momentum", lattice="4x4", n_up=5, n_down=5, u=8.0,
             prec="f64", k="0,0"),
        # the batch configuration's mix, fewer instances, on a kept engine
        dict(name="batch_48", kind="batch", count=48, steps=100),
    ]


# lattices of the configurations, tests and serving mix, by rising size
_LATTICES = ["8", "2x4", "3x3", "10", "2x2x2", "12", "3x4", "2x6", "14", "4x4", "16"]


def _dims(text):
    return tuple(int(d) for d in text.split("x"))


def _sites(text):
    return int(np.prod(_dims(text)))


def _states(lattice, nu, nd):
    n = _sites(lattice)
    return math.comb(n, nu) * math.comb(n, nd)


def _sector(rng, least, most):
    """A sector whose size is spread over the logarithm of [least, most]."""
    want = math.exp(rng.uniform(math.log(least), math.log(most)))
    best = None
    for _ in range(400):
        lat = rng.choice(_LATTICES)
        n = _sites(lat)
        nu = rng.randint(1, n - 1)
        nd = max(1, min(n - 1, nu + rng.choice([0, 0, 0, -1, 1, -2])))
        d = _states(lat, nu, nd)
        if not least <= d <= most:
            continue
        off = abs(math.log(d / want))
        if best is None or off < best[0]:
            best = (off, lat, nu, nd)
        if off < 0.2:
            break
    return dict(lattice=best[1], n_up=best[2], n_down=best[3])


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "host", "ground", "ground", "evolve", "moments",
                       "momentum", "batch"])
    u = round(rng.uniform(0.5, 10.0), 2)
    if kind == "apply":
        prec = rng.choice(["f64", "f64", "f32", "q64"])
        c = dict(kind=kind, u=u, prec=prec, **_sector(rng, 2500, 64e6))
        affine = prec != "q64" and rng.random() < 0.4
        order = "tensor" if prec == "q64" else rng.choice(["reference", "tensor"])
        c.update(order=order, affine=affine)
        return c
    if kind == "host":
        return dict(kind=kind, u=u, prec=rng.choice(["f64", "f64", "f32", "q64"]),
                    **_sector(rng, 5e4, 20e6))
    if kind == "ground":
        if rng.random() < 0.3:
            return dict(kind=kind, u=u, prec="f32", steps=rng.randint(24, 36), refine=True,
                        **_sector(rng, 2e5, 19.1e6))
        return dict(kind=kind, u=u, prec="f64", steps=rng.randint(24, 50), refine=False,
                    **_sector(rng, 3e4, 4e6))
    if kind == "evolve":
        return dict(kind=kind, u=u, prec=rng.choice(["f64", "f64", "q64"]),
                    time=round(rng.uniform(0.1, 0.4), 2),
                    order=rng.choice(["reference", "tensor"]), **_sector(rng, 4e3, 4e6))
    if kind == "moments":
        return dict(kind=kind, u=u, prec=rng.choice(["f64", "q64"]),
                    moments=rng.choice([64, 100, 128]), **_sector(rng, 4e3, 3.4e6))
    if kind == "momentum":
        lat, nu, nd = rng.choice([("4x4", 4, 4), ("4x4", 5, 5), ("4x4", 4, 3), ("4x4", 3, 3),
                                  ("3x4", 5, 5), ("3x4", 6, 6), ("12", 6, 6), ("14", 5, 5)])
        k = ",".join(str(rng.randrange(d)) for d in _dims(lat))
        return dict(kind=kind, lattice=lat, n_up=nu, n_down=nd, u=u,
                    prec=rng.choice(["f64", "f64", "f32", "q64"]), k=k)
    return dict(kind=kind, count=rng.randint(8, 48), steps=rng.randint(80, 100))


# ---------------------------------------------------------------------------
# a user's program
# ---------------------------------------------------------------------------
def _basis(case):
    nu, nd = case["n_up"], case["n_down"]
    return mb.FermionBasis.with_fixed_particle_number_and_spin(_sites(case["lattice"]), nu + nd,
                                                               nu - nd)


def _model(case):
    dims = _dims(case["lattice"])
    make = {1: mb.HubbardModel, 2: mb.HubbardModel2D, 3: mb.HubbardModel3D}[len(dims)]
    return make(1.0, case["u"], *dims)


def _vector(n, seed, dtype=torch.complex128):
    """Uniform on [-1, 1), real and imaginary part: the solvers' start vectors."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    v = torch.rand(2 * n, generator=g, device="cuda", dtype=real)
    v.mul_(2.0).sub_(1.0)
    return torch.view_as_complex(v.view(n, 2))


_AFFINE = dict(scale=0.125, shift=3.0, beta=-1.0)


def _bounds(case):
    """A bracket of the spectrum: each particle's band edges, and U on every pair."""
    nu, nd = case["n_up"], case["n_down"]
    z = 2.0 * len(_dims(case["lattice"]))
    return -z * (nu + nd), z * (nu + nd) + case["u"] * min(nu, nd)


def _batch(case, seed):
    """1D rings of 8, 10 and 12 sites at and next to half filling, U on (0, 8)."""
    rng = np.random.default_rng(int(seed))
    out = []
    for _ in range(case["count"]):
        L = int(rng.choice([8, 10, 12]))
        n = int(rng.choice([L // 2 - 1, L // 2]))
        out.append((L, n, float(rng.uniform(0.5, 8.0)), int(rng.integers(1 << 30))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=int(seed))
    if kind == "batch":
        s["sectors"] = _batch(case, seed)
        s["descs"] = [mb.sector((L,), n, n, 1.0, u) for L, n, u, _ in s["sectors"]]
        s["seeds"] = [sd for *_, sd in s["sectors"]]
        s["engine"] = mb.Engine()
        return s
    dims = _dims(case["lattice"])
    if kind == "momentum":
        nu, nd = case["n_up"], case["n_down"]
        b = mb.FermionBasis.with_fixed_particle_number_spin_momentum(
            _sites(case["lattice"]), nu + nd, nu - nd, dims,
            tuple(int(k) for k in case["k"].split(",")))
        op = mb.GpuHubbardOperator(b, mb.HubbardModelMomentum(1.0, case["u"], dims),
                                   PREC[case["prec"]])
    else:
        op = mb.GpuHubbardOperator(_basis(case), _model(case), PREC[case["prec"]])
    s["op"] = op
    if kind == "moments":
        return s
    x = _vector(op.dimension(), seed, op.dtype)
    if kind == "apply" and case["prec"] == "q64":
        s["x"], s["e"] = op.q64_from_f64(x, order=mb.ORDER_TENSOR)
        s["y"] = op.q64_empty()
    elif kind == "host":
        s["x"] = torch.empty(op.dimension(), dtype=op.dtype, pin_memory=True)
        s["x"].copy_(x)
        s["y"] = torch.empty(op.dimension(), dtype=op.dtype, pin_memory=True)
    else:
        s["x"] = x
        s["y"] = op.empty()
        if case.get("affine"):
            s["z"] = _vector(op.dimension(), seed + 7919, op.dtype)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        r = mb.batch_ground_states(state["descs"], state["seeds"], kmax=case["steps"],
                                   engine=state["engine"])
        # the raw energies come from complex64 vectors
        return dict(e0=np.array([g.e0 for g in r]),
                    e0_raw=np.array([g.e0_raw for g in r], np.float32))
    op = state["op"]
    if kind == "apply":
        if case["prec"] == "q64":
            y, e = op.apply_q64(state["x"], state["e"], out=state["y"])
            return dict(y=y, exponent=e)
        order = ORDER[case["order"]]
        if case["affine"]:
            return op.apply_affine(state["x"], z=state["z"], out=state["y"], order=order, **_AFFINE)
        return op.apply(state["x"], out=state["y"], order=order)
    if kind == "host":
        return op.apply_host(state["x"], state["y"])
    if kind == "ground":
        r = mb.find_min_eigenpair(op, case["steps"], state["x"], refine=case["refine"])
        return dict(value=r.value, steps=r.steps, vector=r.vector)
    if kind == "evolve":
        return mb.time_evolve_state(op, state["x"], case["time"], order=ORDER[case["order"]],
                                    out=state["y"])
    if kind == "moments":
        lo, hi = _bounds(case)
        return mb.kpm_dos_moments(op, case["moments"], 1, state["seed"], lo, hi)
    return op.apply(state["x"], out=state["y"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _hops(case):
    """Mean hops of a state, both spins."""
    dims, n = _dims(case["lattice"]), _sites(case["lattice"])
    bonds = n * len(dims)
    return sum(bonds * 2.0 * k * (n - k) / (n * (n - 1)) for k in (case["n_up"], case["n_down"]))


def _sector_work(dim, hops, size, vectors, applies):
    """`vectors` passes over a vector, `applies` applications of H (one add a
    component and hop, a multiply-add and the diagonal)."""
    return {"bytes": float(vectors) * size * dim, "flops": applies * dim * (2.0 * hops + 6.0)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for L, n in ((8, 3), (8, 4), (10, 4), (10, 5), (12, 5), (12, 6)):  # the mix's mean
            c = dict(lattice=str(L), n_up=n, n_down=n)
            d = _states(str(L), n, n)
            w = _sector_work(d, _hops(c), 8, 5 * case["steps"], case["steps"])
            for k in total:
                total[k] += w[k] * case["count"] / 6.0
        return total
    size = 8 if case["prec"] == "f32" else 16
    dim = _states(case["lattice"], case["n_up"], case["n_down"])
    if kind == "momentum":
        n, nu, nd = _sites(case["lattice"]), case["n_up"], case["n_down"]
        dim //= n
        # one entry a (q, k1, k2) with both targets empty, one int32 each
        row = (n - 1) * nu * nd * ((n - nu) / (n - 1.0)) * ((n - nd) / (n - 1.0))
        return {"bytes": dim * (2.0 * size + 16 + 4 * row), "flops": dim * (2.0 * row + 6.0)}
    hops = _hops(case)
    if kind in ("apply", "host"):
        return _sector_work(dim, hops, size, 3 if case.get("affine") else 2, 1)
    if kind == "moments":
        # a Chebyshev step reads two vectors and writes one
        return _sector_work(dim, hops, size, 3 * (case["moments"] // 2), case["moments"] // 2)
    steps = case.get("steps", 30)
    # a Lanczos step reads v, v_prev and writes the next vector (twice, as alpha
    # is known only after w); the Ritz vector reads every Lanczos vector
    return _sector_work(dim, hops, size, 6 * steps, steps)


# ---------------------------------------------------------------------------
# the same in 64 bits, restated with torch
# ---------------------------------------------------------------------------
def _masks(n, k, dev):
    m = torch.arange(1 << n, dtype=torch.int64, device=dev)
    return m[_count(m, n) == k]


def _count(m, n):
    c = torch.zeros_like(m)
    for i in range(n):
        c += (m >> i) & 1
    return c


def _bonds(dims):
    """{(a, b): multiplicity} of the periodic lattice, first dimension fastest."""
    out = {}
    stride = 1
    n = int(np.prod(dims))
    for d in dims:
        for i in range(n):
            x = (i // stride) % d
            j = i + stride * ((x + 1) % d - x)
            key = (min(i, j), max(i, j))
            out[key] = out.get(key, 0) + 1
        stride *= d
    return out


def _hop_lists(dims, masks):
    """Per state of one spin, for every bond: the target's index (or 0) and the
    matrix element of -sum c+_a c_b + h.c. (0 where the bond does not hop)."""
    idx, val = [], []
    for (a, b), mult in _bonds(dims).items():
        ba, bb = (masks >> a) & 1, (masks >> b) & 1
        live = ba != bb
        t = masks ^ ((1 << a) | (1 << b))
        between = masks & (((1 << b) - 1) & ~((2 << a) - 1))
        sign = 1 - 2 * (_count(between, int(np.prod(dims))) & 1)
        at = torch.searchsorted(masks, t).clamp(max=masks.numel() - 1)
        idx.append(torch.where(live, at, torch.zeros_like(at)))
        val.append(torch.where(live, -mult * sign, torch.zeros_like(sign)).to(torch.float64))
    return idx, val


class _Exact:
    """H of a (N_up, N_down) sector on tensors of shape (D_up, D_down)."""

    def __init__(self, case, dev="cuda"):
        dims = _dims(case["lattice"])
        n = _sites(case["lattice"])
        self.up, self.dn = _masks(n, case["n_up"], dev), _masks(n, case["n_down"], dev)
        self.iu, self.vu = _hop_lists(dims, self.up)
        self.id, self.vd = _hop_lists(dims, self.dn)
        self.n, self.u = n, case["u"]
        self.shape = (self.up.numel(), self.dn.numel())

    def apply(self, x):
        x = x.view(self.shape)
        y = torch.empty_like(x)
        rows = max(1, (1 << 24) // self.shape[1])
        for r in range(0, self.shape[0], rows):
            s = slice(r, r + rows)
            docc = _count(self.up[s, None] & self.dn[None, :], self.n).to(torch.float64)
            acc = x[s] * (self.u * docc)
            for i, v in zip(self.iu, self.vu):
                acc += x[i[s]] * v[s, None]
            for i, v in zip(self.id, self.vd):
                acc += x[s][:, i] * v[None, :]
            y[s] = acc
        return y.view(-1)

    def reference(self):
        """Tensor index of every reference index: the states sorted by their
        occupied slots (orbital by orbital, up before down), compared by
        (spin, orbital)."""
        return _by_slots(self.up[:, None].expand(self.shape).reshape(-1),
                         self.dn[None, :].expand(self.shape).reshape(-1), self.n)


def _by_slots(up, dn, n):
    at = torch.zeros_like(up)
    keys = [torch.zeros_like(up) for _ in range(-(-2 * n // 12))]  # 12 slots of 5 bits each
    for o in range(n):
        for spin, m in ((0, up), (1, dn)):
            here = ((m >> o) & 1).bool()
            for j, key in enumerate(keys):
                place = 12 * j + 11 - at
                key += torch.where(here & (place >= 0) & (place < 12),
                                   (spin * n + o) << (5 * place.clamp(0, 11)), 0)
            at += here
    order = torch.argsort(keys[-1], stable=True)
    for key in keys[-2::-1]:
        order = order[torch.argsort(key[order], stable=True)]
    return order


def _momentum_exact(case, vector, dev="cuda"):
    """H = sum eps(k) n_k + (U/N) sum_q rho_q,up rho_-q,down on the states of
    one total momentum, sorted as the whole basis is."""
    dims, n = _dims(case["lattice"]), _sites(case["lattice"])
    coord = []
    for k in range(n):
        c, r = [], k
        for d in dims:
            c.append(r % d)
            r //= d
        coord.append(c)

    def flat(c):
        s, out = 1, 0
        for v, d in zip(c, dims):
            out += s * (v % d)
            s *= d
        return out

    def total(m):
        t = [torch.zeros_like(m) for _ in dims]
        for k in range(n):
            for d in range(len(dims)):
                t[d] += ((m >> k) & 1) * coord[k][d]
        return t

    up, dn = _masks(n, case["n_up"], dev), _masks(n, case["n_down"], dev)
    tu, td = total(up), total(dn)
    keep = torch.ones(up.numel(), dn.numel(), dtype=torch.bool, device=dev)
    for d, k in enumerate(int(v) for v in case["k"].split(",")):
        keep &= (tu[d][:, None] + td[d][None, :]) % dims[d] == k % dims[d]
    iu, idn = keep.nonzero(as_tuple=True)
    up, dn = up[iu], dn[idn]
    order = _by_slots(up, dn, n)
    up, dn = up[order], dn[order]
    x = vector(up.numel())
    key = (up << n) | dn
    skey, place = torch.sort(key)
    eps = [-2.0 * sum(math.cos(2 * math.pi * c / d) for c, d in zip(coord[k], dims))
           for k in range(n)]
    diag = torch.full((up.numel(),), case["u"] / n * case["n_up"] * case["n_down"],
                      dtype=torch.float64, device=dev)
    for k in range(n):
        diag += eps[k] * ((up >> k) & 1).to(torch.float64)
        diag += eps[k] * ((dn >> k) & 1).to(torch.float64)
    y = diag * x

    def parity(m, a, b):
        lo, hi = min(a, b), max(a, b)
        return _count(m & (((1 << hi) - 1) & ~((2 << lo) - 1)), n) & 1

    acc = torch.zeros_like(x)
    for q in range(1, n):
        for k1 in range(n):
            a = flat([s + t for s, t in zip(coord[k1], coord[q])])
            ok = (((up >> k1) & 1) == 1) & (((up >> a) & 1) == 0)
            i = ok.nonzero().view(-1)
            ui, di, pu = up[i], dn[i], parity(up[i], k1, a)
            u2 = ui ^ ((1 << k1) | (1 << a))
            for k2 in range(n):
                b = flat([s - t for s, t in zip(coord[k2], coord[q])])
                j = ((((di >> k2) & 1) == 1) & (((di >> b) & 1) == 0)).nonzero().view(-1)
                if not j.numel():
                    continue
                t = (u2[j] << n) | (di[j] ^ ((1 << k2) | (1 << b)))
                col = place[torch.searchsorted(skey, t)]
                sign = (1 - 2 * (pu[j] ^ parity(di[j], k2, b))).to(torch.float64)
                acc.index_add_(0, i[j], x[col] * sign)
    return y + case["u"] / n * acc


def _lanczos(h, x, steps):
    """The lowest Ritz value of `steps` Lanczos steps, fully re-orthogonalised."""
    v = torch.empty(steps, x.numel(), dtype=x.dtype, device=x.device)
    v[0] = x / torch.linalg.norm(x)
    a, b = [], []
    for j in range(steps):
        w = h(v[j])
        a.append(float(torch.vdot(v[j], w).real))
        for _ in range(2):
            w = w - (v[:j + 1].conj() @ w) @ v[:j + 1]
        beta = float(torch.linalg.norm(w))
        if j + 1 == steps or beta < 1e-10:
            break
        b.append(beta)
        v[j + 1] = w / beta
    t = np.diag(a) + np.diag(b[:len(a) - 1], 1) + np.diag(b[:len(a) - 1], -1)
    return float(np.linalg.eigvalsh(t)[0])


def _phases(n, seed, stream, dev):
    """exp(2 pi i u), u from the Philox4x32-10 block of (index, stream, seed)."""
    lo = (1 << 32) - 1
    i = torch.arange(n, dtype=torch.int64, device=dev)
    c = [i & lo, i >> 32, torch.full_like(i, stream), torch.zeros_like(i)]
    k = [seed & lo, seed >> 32]

    def mul(m, v):
        p0, p1 = m * (v & 0xFFFF), m * (v >> 16)
        s = (p1 & 0xFFFF_FFFF_FFFF) + (p0 >> 16)
        return (s >> 16) & lo, ((s << 16) | (p0 & 0xFFFF)) & lo

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k[0], l1, h0 ^ c[3] ^ k[1], l0]
        k = [(k[0] + 0x9E3779B9) & lo, (k[1] + 0xBB67AE85) & lo]
    u = ((c[0] << 20) | (c[1] >> 12)).to(torch.float64) * 2.0 ** -52
    return torch.polar(torch.ones_like(u), 2.0 * math.pi * u)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        e = []
        for L, n, u, sd in _batch(case, seed):
            h = _Exact(dict(lattice=str(L), n_up=n, n_down=n, u=u))
            e.append(_lanczos(h.apply, _vector(h.shape[0] * h.shape[1], sd), 80))
        return dict(e0=np.array(e), e0_raw=None)
    if kind == "momentum":
        dt = torch.complex64 if case["prec"] == "f32" else torch.complex128
        return _momentum_exact(case, lambda n: _vector(n, seed, dt).to(torch.complex128)).cpu()
    h = _Exact(case)
    dim = h.shape[0] * h.shape[1]
    if kind == "moments":
        lo, hi = _bounds(case)
        a, b = (hi - lo) / 2.0 * 1.01, (hi + lo) / 2.0
        t0 = _phases(dim, int(seed), 1, "cuda")
        t1 = (h.apply(t0) - b * t0) / a
        r = t0
        mu = [dim, float(torch.vdot(r, t1).real)]
        base0, base1 = mu
        while len(mu) < case["moments"]:
            s = len(mu) // 2
            mu.append(2.0 * float(torch.vdot(t1, t1).real) - base0)
            t0, t1 = t1, 2.0 * (h.apply(t1) - b * t1) / a - t0
            mu.append(2.0 * float(torch.vdot(t0, t1).real) - base1)
            assert len(mu) == 2 * s + 2
        return np.array(mu[:case["moments"]]) / dim
    dt = torch.complex64 if case["prec"] == "f32" else torch.complex128
    x = _vector(dim, seed, dt).to(torch.complex128)
    if kind == "apply" and case["prec"] == "q64":
        return None  # integers: the same or not
    order = None
    if kind in ("host", "ground") or case.get("order") == "reference":
        order = h.reference()
        t = torch.empty_like(x)
        t[order] = x
        x = t
    back = (lambda y: y[order]) if order is not None else (lambda y: y)
    if kind in ("apply", "host"):
        y = h.apply(x)
        if case.get("affine"):
            z = _vector(dim, seed + 7919, dt).to(torch.complex128)
            if order is not None:
                t = torch.empty_like(z)
                t[order] = z
                z = t
            y = _AFFINE["scale"] * (y - _AFFINE["shift"] * x) + _AFFINE["beta"] * z
        return back(y).cpu()
    if kind == "ground":
        if dim > 5e6:
            return None
        # the Ritz vector's sign is free; the refinement goes on for 8 Krylov steps
        # from the Ritz vector, which no plain run of 64 bits restates
        return None if case["refine"] else dict(value=_lanczos(h.apply, x, case["steps"]),
                                                steps=None, vector=None)
    # exp(-i t H) by Taylor steps of at most unit norm
    lo, hi = _bounds(case)
    steps = max(1, math.ceil(case["time"] * max(abs(lo), abs(hi)) / 2.0))
    dt_ = case["time"] / steps
    for _ in range(steps):
        term, k = x, 1
        while k <= 30:
            term = h.apply(term) * (-1j * dt_ / k)
            x = x + term
            k += 1
    return back(x).cpu()
