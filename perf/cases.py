"""The work this library is measured on: what its users have it do, over the sizes they do it at.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program holds
before the call (a handle with a configuration in it, its pinned host arrays), run() is one pass
through the public entry points, work() the bytes and operations such a pass cannot do without, and
exact() the same results in plain 64-bit torch, without this library.

Configurations: links 1 + s N(0,1)^4, normalised, with s chosen so that the mean plaquette is that of
the beta = 3.09 ensembles (0.73), on top of constant abelian fluxes that give the field a topological
charge of the size found on such lattices, all turned by a random gauge transformation, so that no
link is near 1.  Staples, acceptance rates, loops and charges are then those of a thermalised field.

Results of an FP32 handle are returned as 32-bit numbers, the precision they have.
"""
import ctypes
import math

import numpy as np
import torch

from masterarbeit_b200 import Lattice
from masterarbeit_b200.su2g import APE, Batch, load

BETA = 3.09
NOISE = 0.23


# ------------------------------------------------------------------- cases ---

def listed():
    return [
        # The update program on the smallest production test lattice: 20 heatbath sweeps with the
        # plaquette after each, then the configuration is fetched to be written.  Launch latency.
        dict(name="qcd_8_f64", kind="qcd", t=8, x=8, y=8, z=8, sweeps=20),
        # The same on the lattice of the thesis' thermalisation runs.
        dict(name="qcd_24_f64", kind="qcd", t=24, x=24, y=24, z=24, sweeps=20),
        # The production lattice of the benchmark, in the reference's precision.
        dict(name="qcd_48_f64", kind="qcd", t=48, x=48, y=48, z=48, sweeps=30),
        # Thermalisation with four unsmeared loops logged after every sweep (the Therm runs), on an
        # uneven lattice.
        dict(name="therm_f64", kind="therm", t=24, x=14, y=18, z=22, sweeps=4),
        # The mixed update, one heatbath and four overrelaxation sweeps, in FP32 on an uneven lattice.
        dict(name="mixed_f32", kind="mixed", t=40, x=30, y=36, z=34, sweeps=2),
        # Many small chains at once, FP32, mixed update, plaquette after every sweep.
        dict(name="batch_64x12_f32", kind="batch", replicas=64, t=12, x=12, y=12, z=12, sweeps=2),
        # One configuration of the loop and charge measurement in FP32 on the production lattice.
        dict(name="meas_48_f32", kind="meas", f32=True, t=48, x=48, y=48, z=48, n_q=30, n_s=100, r=9, tt=9),
        # The same in the reference's precision on the smaller production lattice.
        dict(name="meas_24_f64", kind="meas", f32=False, t=24, x=24, y=24, z=24, n_q=30, n_s=100, r=9, tt=9),
        # The charge program: read a configuration, then Q after every APE step (20 of them), and the
        # smeared field back.
        dict(name="qtop_f64", kind="qtop", t=16, x=12, y=10, z=14, steps=20),
        # The gradient of the smeared charge, as an optimiser calls it: FP32 after few steps (the more
        # steps, the more of the gradient is the rounding of its cancelling terms), FP64 after more.
        dict(name="vjp_24_f32", kind="vjp", f32=True, t=24, x=24, y=24, z=24, n_ape=3),
        dict(name="vjp_f64", kind="vjp", f32=False, t=16, x=12, y=16, z=20, n_ape=10),
        # Smearing a device field that another component owns (no allocation), spatial links.
        dict(name="inplace_f64", kind="inplace", t=20, x=16, y=18, z=14, steps=20, mode="spatial"),
    ]


def _extents(rng, lo, hi):
    """Four even extents of geometric mean between lo and hi (uniform in its logarithm), unequal."""
    m = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    e = [max(4, 2 * round(0.5 * m * math.exp(rng.uniform(-0.3, 0.3)))) for _ in range(4)]
    while math.prod(e) > hi ** 4:
        e[e.index(max(e))] -= 2
    return dict(zip("txyz", e))


def draw(rng):
    kind = rng.choice(["qcd", "therm", "mixed", "batch", "meas", "qtop", "vjp", "inplace"])
    if kind == "qcd":
        return dict(kind=kind, sweeps=rng.randint(5, 25), **_extents(rng, 8, 46))
    if kind == "therm":
        return dict(kind=kind, sweeps=rng.randint(1, 6), **_time_in_eights(_extents(rng, 10, 30)))
    if kind == "mixed":
        return dict(kind=kind, sweeps=rng.randint(1, 2), **_extents(rng, 10, 46))
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(4, 64), sweeps=2, **_extents(rng, 6, 14))
    if kind == "meas":
        f32 = rng.random() < 0.5
        e = _extents(rng, 12, 44) if f32 else _time_in_eights(_extents(rng, 12, 30))
        return dict(kind=kind, f32=f32, n_q=rng.randint(5, 30), n_s=rng.randint(20, 100), r=rng.randint(3, 10),
                    tt=rng.randint(3, min(12, e["t"] - 1)), **e)
    if kind == "qtop":
        return dict(kind=kind, steps=rng.randint(5, 20), **_extents(rng, 8, 24))
    if kind == "vjp":
        f32 = rng.random() < 0.5
        return dict(kind=kind, f32=f32, n_ape=rng.randint(1, 3) if f32 else rng.randint(5, 30),
                    **_extents(rng, 8, 24 if f32 else 18))
    return dict(kind=kind, steps=rng.randint(5, 30), mode=rng.choice(["all", "spatial", "temporal"]),
                **_extents(rng, 8, 22))


def _time_in_eights(e):
    """FP64 loops of R >= 4 are measured at time extents like the production lattices', multiples of 8."""
    return dict(e, t=max(8, 8 * (e["t"] // 8)))


def _dims(case):
    return tuple(case[k] for k in "txyz")


def _therm_loops():
    return [1, 1, 5, 5], [1, 5, 1, 5]   # W(1,1), W(1,5), W(5,1), W(5,5)


def _grid(case):
    pairs = [(r, t) for r in range(1, case["r"] + 1) for t in range(1, case["tt"] + 1)]
    return [p[0] for p in pairs], [p[1] for p in pairs]


# ------------------------------------------------------------ configurations ---

def _mul(a, b):
    """Quaternion product; component first: (4, ...)."""
    a0, a1, a2, a3 = a
    b0, b1, b2, b3 = b
    return torch.stack((a0 * b0 - a1 * b1 - a2 * b2 - a3 * b3, a0 * b1 + a1 * b0 - a2 * b3 + a3 * b2,
                        a0 * b2 + a1 * b3 + a2 * b0 - a3 * b1, a0 * b3 - a1 * b2 + a2 * b1 + a3 * b0))


def _dag(a):
    return torch.stack((a[0], -a[1], -a[2], -a[3]))


def _up(a, mu, k=1):
    """The field at x + k mu."""
    return torch.roll(a, -k, dims=1 + mu)


def _unit(a):
    return a / torch.sqrt((a * a).sum(0, keepdim=True))


def _configuration(dims, seed, f32=False):
    """Four links fields of shape (4, T, X, Y, Z), 64 bits, on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    opt = dict(device="cuda", dtype=torch.float64)
    g = _unit(torch.randn((4, *dims), generator=gen, **opt))
    out = []
    at = [torch.arange(n, **opt).reshape([-1 if d == i else 1 for i in range(4)]) for d, n in enumerate(dims)]
    for mu in range(4):
        u = NOISE * torch.randn((4, *dims), generator=gen, **opt)
        u[0] += 1.0
        u = _unit(u)
        # constant flux 2 pi n / (L_a L_b) through the planes (0, 1) and (2, 3): charge 2 n^2
        a, b = (0, 1) if mu < 2 else (2, 3)
        unit = 2.0 * math.pi * (2 if dims[a] * dims[b] >= 256 else 1)
        angle = torch.zeros(dims, **opt)
        if mu == b:
            angle = angle + unit / (dims[a] * dims[b]) * at[a]
        else:
            angle = angle - unit / dims[b] * at[b] * (at[a] == dims[a] - 1)
        zero = torch.zeros_like(angle)
        u = _mul(u, torch.stack((torch.cos(angle), zero, zero, torch.sin(angle))))
        u = _mul(_mul(g, u), _dag(_up(g, mu)))
        out.append(u.float().double() if f32 else u)
    return out


def _to_host_layout(links):
    """(V, 4 directions, 4 components), the layout of the host arrays."""
    return torch.stack(links, 0).reshape(4, 4, -1).permute(2, 0, 1).contiguous()


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


# --------------------------------------------------------------- the passes ---

def prepare(case, seed):
    kind, dims = case["kind"], _dims(case)
    s = dict(case=case)
    if kind == "inplace":
        s["field"] = _to_host_layout(_configuration(dims, seed))
        s["dims"] = (ctypes.c_int32 * 4)(*dims)
        s["lib"] = load()
        return s
    if kind == "batch":
        s["batch"] = Batch([dict(dims=dims, beta=BETA, seed=seed * 1000 + i, replica=i, start="cold")
                            for i in range(case["replicas"])], precision="fp32")
        for i in range(case["replicas"]):
            s["batch"].upload(i, _to_host_layout(_configuration(dims, seed * 1000 + i)).cpu().numpy())
        return s
    f32 = kind == "mixed" or case.get("f32", False)
    s["lat"] = Lattice(dims, precision="fp32" if f32 else "fp64", beta=BETA, seed=seed, start="cold")
    links = _to_host_layout(_configuration(dims, seed)).cpu().numpy()
    if kind == "qtop":
        s["links"] = _pinned(*links.shape).copy_(torch.from_numpy(links))
    else:
        s["lat"].upload(links)
    if kind in ("qcd", "therm", "qtop"):
        s["host"] = _pinned(*links.shape)
    if kind == "vjp":
        s["grad"] = _pinned(links.shape[0], 4, 3)
    return s


def run(s):
    case = s["case"]
    return _RUN[case["kind"]](s, case)


def _run_qcd(s, case):
    """The update program between two configurations: sweeps with a plaquette each, then the field."""
    plaq, acc = s["lat"].graph_run(case["sweeps"], 1, 1, 0)
    s["lat"].download(s["host"].numpy())
    return dict(plaq=plaq, acc=acc, links=s["host"])


def _run_therm(s, case):
    """Thermalisation, call by call: a sweep with its plaquette, then the four logged loops."""
    R, T = _therm_loops()
    plaq, loops = [], []
    for _ in range(case["sweeps"]):
        plaq.append(s["lat"].sweep_plaquette(1, 1, 0))
        loops.append(s["lat"].wilson(R, T))
    s["lat"].download(s["host"].numpy())
    return dict(plaq=np.array(plaq), loops=np.array(loops), links=s["host"])


def _run_mixed(s, case):
    """One heatbath and four overrelaxation sweeps, in FP32; what the call returns.  (Two FP32 fields
    that differ in a rounding draw differently wherever an accept test lies between them.)"""
    plaq, acc = s["lat"].sweep_plaquette(case["sweeps"], 1, 4, acc=True)
    return dict(plaq=np.float32(plaq), acc=np.float32(acc))


def _run_batch(s, case):
    return s["batch"].run(case["sweeps"], 1, 4, 1)[0].astype(np.float32)


def _run_meas(s, case):
    """One configuration: Q at half and at all of the APE steps, W(R, T) after spatial smearing."""
    R, T = _grid(case)
    n = case["n_q"]
    q, w = s["lat"].measure(q_ape=[n - n // 2, n], alpha_q=0.5, R=R, T=T, ns_s=case["n_s"], alpha_s=0.5)
    return dict(q=q.astype(np.float32), w=w.astype(np.float32)) if case["f32"] else dict(q=q, w=w)


def _run_qtop(s, case):
    """Read a configuration, Q (and its sum of absolute values) after every APE step, field back."""
    lat, q = s["lat"], []
    lat.upload(s["links"].numpy())
    for _ in range(case["steps"]):
        lat.ape(1, 0.5, "all")
        q.append(lat.qtop(with_abs=True))
    lat.download(s["host"].numpy())
    return dict(q=np.array(q), links=s["host"])


def _run_vjp(s, case):
    """Q after the smearing and its gradient into a pinned host array (the C call)."""
    lat, q = s["lat"], ctypes.c_double()
    grad = ctypes.cast(s["grad"].data_ptr(), ctypes.POINTER(ctypes.c_double))
    lat._check(lat.lib.su2g_ape_qtop_vjp(lat.h, case["n_ape"], 0.5, 0, ctypes.byref(q), grad))
    if case["f32"]:
        return dict(q=np.float32(q.value), grad=s["grad"].float())
    return dict(q=np.float64(q.value), grad=s["grad"])


def _run_inplace(s, case):
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = s["lib"].su2g_ape_inplace_noalloc(ctypes.c_void_p(s["field"].data_ptr()), s["dims"], case["steps"], 0.5,
                                           APE[case["mode"]], stream)
    if rc:
        raise RuntimeError(s["lib"].su2g_last_error(None).decode())
    return s["field"]


_RUN = dict(qcd=_run_qcd, therm=_run_therm, mixed=_run_mixed, batch=_run_batch, meas=_run_meas, qtop=_run_qtop,
            vjp=_run_vjp, inplace=_run_inplace)


# ------------------------------------------------------------------- floors ---

_MUL = 28   # flops of one quaternion product


def _sweep_work(V, size, n=1.0):
    """A sweep over all links: eight passes, each reading the 3V links of the other directions and the
    V/2 of the other parity and writing V/2; twelve products for a staple sum, about four to draw."""
    return dict(bytes=n * 8 * 4 * V * size, flops=n * 4 * V * 16 * _MUL)


def _ape_work(V, size, mode, n):
    """One step: every link the staples need read once, the smeared ones written."""
    read, written, staples = {"all": (4, 4, 24), "spatial": (3, 3, 12), "temporal": (4, 1, 6)}[mode]
    return dict(bytes=n * (read + written) * V * size, flops=n * V * staples * 2 * _MUL)


def _charge_work(V, size, n):
    """Six planes, three clover sizes, four leaves of four segments each."""
    return dict(bytes=n * 4 * V * size, flops=n * V * (8 + 6 * 3 * 4 * 3) * _MUL)


def _loop_work(V, size, r, t):
    """Line products: for each R and spatial direction the transported line, two products per T."""
    return dict(bytes=4 * V * size, flops=V * 3 * r * (1 + 2 * t) * _MUL)


def work(case):
    kind, V = case["kind"], math.prod(_dims(case))
    size = 16 if kind in ("mixed", "batch") or case.get("f32", False) else 32
    host = 128 * V   # the field in the host layout
    if kind == "qcd":
        parts = [_sweep_work(V, size, case["sweeps"]), dict(bytes=host, flops=0)]
    elif kind == "therm":
        n = case["sweeps"]
        parts = [_sweep_work(V, size, n), dict(bytes=host, flops=0)] + [_loop_work(V, size, 2, 5)] * n
    elif kind == "mixed":
        parts = [_sweep_work(V, size, 5 * case["sweeps"])]
    elif kind == "batch":
        parts = [_sweep_work(V, size, 5 * case["sweeps"] * case["replicas"])]
    elif kind == "meas":
        parts = [_ape_work(V, size, "all", case["n_q"]), _charge_work(V, size, 2),
                 _ape_work(V, size, "spatial", case["n_s"]), _loop_work(V, size, case["r"], case["tt"])]
    elif kind == "qtop":
        parts = [dict(bytes=2 * host, flops=0), _ape_work(V, size, "all", case["steps"]),
                 _charge_work(V, size, case["steps"])]
    elif kind == "vjp":
        # forward; backwards each step reads the field and a gradient and writes one, with three
        # products for each of the forward's factors; the charge and its gradient
        n = case["n_ape"]
        parts = [_ape_work(V, size, "all", n), dict(bytes=n * 12 * V * size, flops=n * V * 4 * 30 * _MUL),
                 _charge_work(V, size, 3), dict(bytes=96 * V, flops=0)]
    else:
        parts = [_ape_work(V, size, case["mode"], case["steps"])]
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


# -------------------------------------------------------- 64-bit references ---

def _staple(U, mu, directions):
    """S_mu(x) = sum_nu U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu)."""
    S = torch.zeros_like(U[mu])
    for nu in directions:
        if nu == mu:
            continue
        side = _up(U[nu], mu)
        S = S + _mul(_mul(U[nu], _up(U[mu], nu)), _dag(side))
        S = S + _up(_mul(_mul(_dag(U[nu]), U[mu]), side), nu, -1)
    return S


def _ape(U, mode, alpha=0.5):
    change = {"all": range(4), "spatial": range(1, 4), "temporal": range(1)}[mode]
    around = range(4) if mode == "all" else range(1, 4)
    return [_unit(U[mu] + alpha * _staple(U, mu, around)) if mu in change else U[mu] for mu in range(4)]


def _plaquette(U):
    total = sum((_mul(U[a], _up(U[b], a)) * _mul(U[b], _up(U[a], b))).sum() for a in range(4) for b in range(a + 1, 4))
    return (total / (6 * U[0][0].numel())).item()


def _charge_density(U):
    """8 [tr F01 F23 + tr F02 F31 + tr F03 F12] of the improved clover field strength."""
    F = {}
    lines = {1: U}
    for e in (2, 3):
        lines[e] = [_mul(lines[e - 1][d], _up(U[d], d, e - 1)) for d in range(4)]
    for a, b in ((0, 1), (2, 3), (0, 2), (3, 1), (0, 3), (1, 2)):
        f = 0
        for e, k in ((1, 1.5), (2, -0.15), (3, 1.0 / 90.0)):
            A, B = lines[e][a], lines[e][b]
            ab, ba = _mul(A, _up(B, a, e)), _mul(B, _up(A, b, e))   # x -> x + a + b by both ways
            leaf = _mul(ab, _dag(ba))
            leaf = leaf + _mul(_up(_mul(_dag(B), ab), b, -e), _dag(A))
            leaf = leaf + _mul(B, _up(_mul(_dag(ba), A), a, -e))
            leaf = leaf + _up(_up(_mul(_dag(ba), ab), a, -e), b, -e)
            f = f + 0.25 * k * leaf[1:]
        F[a, b] = f
    return -16 * sum((F[p] * F[q]).sum(0) for p, q in (((0, 1), (2, 3)), ((0, 2), (3, 1)), ((0, 3), (1, 2))))


def _charge(U):
    d = _charge_density(U) / (32 * math.pi ** 2)
    return d.sum().item(), d.abs().sum().item()


def _loops(U, R, T):
    found = {}
    time = {}
    line = None
    for t in range(1, max(T) + 1):
        line = U[0] if t == 1 else _mul(line, _up(U[0], 0, t - 1))
        if t in T:
            time[t] = line
    for k in range(1, 4):
        line = None
        for r in range(1, max(R) + 1):
            line = U[k] if r == 1 else _mul(line, _up(U[k], k, r - 1))
            for t in {tt for rr, tt in zip(R, T) if rr == r}:
                w = (_mul(time[t], _up(line, 0, t)) * _mul(line, _up(time[t], k, r))).sum().item()
                found[r, t] = found.get((r, t), 0.0) + w / (3 * U[0][0].numel())
    return np.array([found[p] for p in zip(R, T)])


def _philox(counter, key):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors of 32-bit words."""
    m = 0xFFFFFFFF
    x, y, z, w = counter
    k0, k1 = key
    for _ in range(10):
        p, q = x * 0xD2511F53, z * 0xCD9E8D57
        x, y, z, w = ((q >> 32) & m) ^ y ^ k0, q & m, ((p >> 32) & m) ^ w ^ k1, p & m
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return [(v.double() + 0.5) / 4294967296.0 for v in (x, y, z, w)]


def _heatbath_sweep(U, beta, seed, sweep):
    """One checkerboard heatbath sweep in place; the mean of 1/trials."""
    dims = tuple(U[0].shape[1:])
    at = torch.meshgrid(*[torch.arange(n, device="cuda") for n in dims], indexing="ij")
    site = ((at[0] * dims[1] + at[1]) * dims[2] + at[2]) * dims[3] + at[3]
    parity = (at[0] + at[1] + at[2] + at[3]) & 1
    key = (seed & 0xFFFFFFFF, seed >> 32)
    accepted = 0.0
    for mu in range(4):
        for par in range(2):
            here = parity == par
            A = _dag(_staple(U, mu, range(4)))[:, here]
            n = site[here]
            norm = torch.sqrt((A * A).sum(0))

            def words(draw, tag, which):
                full = torch.full_like(n[which], (draw << 3) | (mu << 1) | tag)
                return _philox((n[which], torch.full_like(full, sweep), full, torch.zeros_like(full)), key)

            delta = torch.zeros_like(norm)
            trials = torch.zeros_like(norm)
            left = torch.arange(norm.numel(), device="cuda")
            trial = 0
            while left.numel():
                u0, u1, u2, u3 = words(trial, 0, left)
                d = -(torch.log(u1) + torch.log(u0) * torch.cos(2 * math.pi * u2) ** 2) / (beta * norm[left])
                ok = u3 * u3 <= 1 - 0.5 * d
                trial += 1
                delta[left[ok]] = d[ok]
                trials[left[ok]] = trial
                left = left[~ok]
            a0, a1, _, _ = words(0, 1, torch.arange(norm.numel(), device="cuda"))
            s = torch.sqrt(delta * (2 - delta))
            st = 2 * torch.sqrt(a1 * (1 - a1))
            X = torch.stack((1 - delta, s * st * torch.cos(2 * math.pi * a0), s * st * torch.sin(2 * math.pi * a0),
                             s * (1 - 2 * a1)))
            U[mu][:, here] = _mul(X, _dag(A / norm))
            accepted += (1.0 / trials).sum().item()
    return accepted / (4 * U[0][0].numel())


def _gradient(U, n_ape):
    """Q after n_ape steps and the su(2) gradient of every link, by automatic differentiation."""
    from torch.utils.checkpoint import checkpoint
    leaf = [u.clone().requires_grad_(True) for u in U]
    V = leaf
    for _ in range(n_ape):
        V = checkpoint(lambda *u: tuple(_ape(list(u), "all")), *V, use_reentrant=False)
    Q = checkpoint(lambda *u: _charge_density(list(u)).sum(), *V, use_reentrant=False) / (32 * math.pi ** 2)
    Q.backward()
    g = [_mul(u.grad, _dag(u.detach()))[1:] for u in leaf]
    return Q.item(), torch.stack(g, 0).reshape(4, 3, -1).permute(2, 0, 1).contiguous()


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    if kind in ("mixed", "batch"):
        return None   # an FP32 accept test near its threshold decides by rounding: no 64-bit value
    U = _configuration(dims, seed, f32=case.get("f32", False))
    if kind == "inplace":
        for _ in range(case["steps"]):
            U = _ape(U, case["mode"])
        return _to_host_layout(U)
    if kind in ("qcd", "therm"):
        plaq, acc, loops = [], [], []
        for k in range(case["sweeps"]):
            acc.append(_heatbath_sweep(U, BETA, seed, k))
            plaq.append(_plaquette(U))
            if kind == "therm":
                loops.append(_loops(U, *_therm_loops()))
        links = _to_host_layout(U).cpu()
        if kind == "therm":
            return dict(plaq=np.array(plaq), loops=np.array(loops), links=links)
        return dict(plaq=np.array(plaq), acc=np.array(acc), links=links)
    if kind == "meas":
        n, W, q = case["n_q"], U, []
        for k in range(n):
            W = _ape(W, "all")
            if k + 1 in (n - n // 2, n):
                q.append(_charge(W)[0])
        for _ in range(case["n_s"]):
            U = _ape(U, "spatial")
        return dict(q=np.array(q), w=_loops(U, *_grid(case)))
    if kind == "qtop":
        q = []
        for _ in range(case["steps"]):
            U = _ape(U, "all")
            q.append(_charge(U))
        return dict(q=np.array(q), links=_to_host_layout(U).cpu())
    Q, grad = _gradient(U, case["n_ape"])
    return dict(q=np.float64(Q), grad=grad.cpu())
