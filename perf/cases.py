"""What is timed: the work a user of the library has it do, through its
public entry points (the Python package over the C ABI).

Kinds of case
  pf        one particle filter over a recorded observation sequence, host
            arrays in, histories out (precision 32 or 64)
  batch     many independent filters of uneven sizes and horizons run together
  learned   bearings-only filters with the network proposal
  resample  one resampling of FP64 weights with an engine: replication counts,
            and with select also parent indices and the particle copy
  weight    the Weight class on device (set / set_log / add_log, ESS) and the
            monitor's weighted mean
  rng       bulk random numbers from an engine
  mlp       the proposal network: forward pass, or loss and gradient (the
            inner step of its training)
"""
import ctypes
import math

import numpy as np
import torch

import vsmc_gb300 as vc

SCHEMES = list(vc.SCHEMES)


def listed():
    return [
        # The reference's own pf example: 1000 particles, 100 observations.
        # Launches and latency are all of it.
        {"name": "pf32_n1000", "kind": "pf", "precision": 32, "n": 1000,
         "T": 100, "scheme": "stratified", "threshold": 0.5},
        # An ordinary tracking filter of a size nobody rounded.
        {"name": "pf32_n100003", "kind": "pf", "precision": 32, "n": 100003,
         "T": 100, "scheme": "systematic", "threshold": 0.5},
        # The headline benchmark's filter, with a shorter horizon.
        {"name": "pf32_n16777216", "kind": "pf", "precision": 32,
         "n": 1 << 24, "T": 50, "scheme": "systematic", "threshold": 0.5},
        # The reference's arithmetic step for step (validation runs): the
        # 64-seed parity configuration.
        {"name": "pf64_n16384", "kind": "pf", "precision": 64, "n": 1 << 14,
         "T": 100, "scheme": "stratified", "threshold": 0.5},
        # Many trackers at once, sizes and horizons uneven as in the batched
        # benchmark.
        {"name": "batch_512", "kind": "batch", "nf": 512, "nmin": 256,
         "nmax": 65536, "Tmin": 20, "Tmax": 120, "scheme": "stratified"},
        # Filters with the trained proposal.
        {"name": "learned_64x4096", "kind": "learned", "nf": 64, "n": 4096,
         "T": 50, "scheme": "systematic"},
        # One resampling of a small population: latency.
        {"name": "resample_systematic_1000", "kind": "resample", "n": 1000,
         "scheme": "systematic", "select": False, "sd": 1.0},
        # One resampling of a very large population (the resampling
        # microbenchmark's size and weights).
        {"name": "resample_stratified_16777216", "kind": "resample",
         "n": 1 << 24, "scheme": "stratified", "select": False, "sd": 3.0},
        # The whole selection step as a program of its own makes it: counts,
        # parents, copy of the particles; the reference's default scheme at a
        # size that is no power of two.
        {"name": "select_multinomial_1000003", "kind": "resample",
         "n": 1000003, "scheme": "multinomial", "select": True, "sd": 1.0},
        # Log-weights of a million particles to weights, ESS and the
        # weighted mean.
        {"name": "weight_set_log_1048576", "kind": "weight", "n": 1 << 20,
         "op": "set_log", "sd": 3.0},
        # Bulk normals in double precision, an odd number of them.
        {"name": "normal_f64_4194305", "kind": "rng", "n": (1 << 22) + 1,
         "dist": "normal", "bits": 64, "engine": "philox"},
        # One training minibatch of the proposal network.
        {"name": "mlp_grad_65536", "kind": "mlp", "op": "grad",
         "B": 1 << 16},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pf", "pf", "pf", "batch", "learned", "resample",
                       "resample", "weight", "rng", "rng", "mlp"])
    if kind == "pf":
        precision = rng.choice([32, 32, 64])
        if precision == 32:
            n = _logint(rng, 256, 1 << 24)
            T = min(rng.randint(20, 200), max(8, (1 << 29) // n))
            scheme = rng.choice(["stratified", "systematic"])
        else:
            n = _logint(rng, 256, 1 << 17)
            T = rng.randint(20, 100)
            scheme = rng.choice(SCHEMES)
        return {"kind": "pf", "precision": precision, "n": n, "T": T,
                "scheme": scheme, "threshold": rng.choice([0.3, 0.5, 0.8])}
    if kind == "batch":
        nmin = _logint(rng, 64, 512)
        return {"kind": "batch", "nf": _logint(rng, 8, 512), "nmin": nmin,
                "nmax": _logint(rng, 1024, 65536), "Tmin": rng.randint(5, 20),
                "Tmax": rng.randint(30, 120),
                "scheme": rng.choice(["stratified", "systematic"])}
    if kind == "learned":
        return {"kind": "learned", "nf": _logint(rng, 8, 64),
                "n": _logint(rng, 300, 4096), "T": rng.randint(10, 50),
                "scheme": rng.choice(["stratified", "systematic"])}
    if kind == "resample":
        select = rng.random() < 0.5
        return {"kind": "resample", "n": _logint(rng, 200, 1 << 24),
                "scheme": rng.choice(SCHEMES), "select": select,
                "sd": round(rng.uniform(0.5, 3.0), 2)}
    if kind == "weight":
        return {"kind": "weight", "n": _logint(rng, 200, 1 << 22),
                "op": rng.choice(["set", "set_log", "add_log"]),
                "sd": round(rng.uniform(0.5, 3.0), 2)}
    if kind == "rng":
        dist = rng.choice(["rand", "u01", "normal", "normal", "student_t"])
        n = _logint(rng, 1000, 1 << (15 if dist == "student_t" else 24))
        return {"kind": "rng", "n": n, "dist": dist,
                "bits": 64 if dist in ("rand", "student_t")
                else rng.choice([32, 64]),
                "engine": rng.choice(["philox", "philox", "threefry"])}
    op = rng.choice(["grad", "forward"])
    return {"kind": "mlp", "op": op, "B": _logint(rng, 100, 1 << 18)}


# ------------------------------------------------------------------ inputs


def _simulate(rng, T, m):
    """Observations of the constant-velocity / Student-t model."""
    p = rng.normal(0, m.sd_pos0, 2)
    v = rng.normal(0, m.sd_vel0, 2)
    obs = np.empty((T, 2))
    for t in range(T):
        if t:
            a = rng.normal(0, m.sigma_a, 2)
            p = p + m.dt * v + 0.5 * m.dt ** 2 * a
            v = v + m.dt * a
        obs[t] = p + m.obs_scale * rng.standard_t(m.nu, 2)
    return obs


def _simulate_bearings(rng, T, m):
    p = np.array([m.x0, m.y0]) + rng.normal(0, m.sd_pos0, 2)
    v = np.array([m.vx0, m.vy0]) + rng.normal(0, m.sd_vel0, 2)
    q = m.q
    L = np.linalg.cholesky(np.array([[q * m.dt ** 3 / 3, q * m.dt ** 2 / 2],
                                     [q * m.dt ** 2 / 2, q * m.dt]]))
    z = np.empty(T)
    for t in range(T):
        if t:
            e = L @ rng.normal(0, 1, (2, 2))
            p, v = p + m.dt * v + e[0], v + e[1]
        z[t] = math.atan2(p[1], p[0]) + rng.normal(0, m.sigma_z)
    return z


def _network(rng):
    """A proposal network with weights of a trained one's size."""
    W = [rng.normal(0, 0.5, (64, 6)), rng.normal(0, 0.1, 64),
         rng.normal(0, 0.15, (64, 64)), rng.normal(0, 0.1, 64),
         rng.normal(0, 0.03, (8, 64)), rng.normal(0, 0.02, 8)]
    return [w.astype(np.float32) for w in W]


def _batch_spec(case):
    """Sizes, horizons and models of a batch: part of the case, as they are
    of a program's configuration; seeds and observations are its inputs."""
    nf = case["nf"]
    rng = np.random.default_rng(nf + case["nmax"])
    n = np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]),
                           nf)).astype(np.uint32)
    T = rng.integers(case["Tmin"], case["Tmax"] + 1, nf).astype(np.uint32)
    models = []
    for _ in range(nf):
        m = vc.default_model()
        m.sigma_a = float(rng.uniform(0.5, 2.0))
        m.obs_scale = float(rng.uniform(0.2, 1.0))
        models.append(m)
    return n, T, models


def _histories(TT):
    return (np.zeros((TT, 2)), np.zeros(TT), np.zeros(TT, np.int32),
            np.zeros(TT))


def _mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    W = _network(rng)
    feat = rng.uniform(-1, 1, (case["B"], 6)).astype(np.float32)
    nu = rng.normal(0, 1, (case["B"], 4)).astype(np.float32)
    return W, feat, nu


def _log_weights(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return case["sd"] * torch.randn(case["n"], dtype=torch.float64,
                                    device="cuda", generator=g)


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "pf":
        rng = np.random.default_rng(seed)
        s["pf"] = vc.ParticleFilter(
            case["n"], case["precision"], vc.SCHEMES[case["scheme"]],
            case["threshold"], seed=seed + 1, max_steps=case["T"])
        s["obs"] = _simulate(rng, case["T"], vc.default_model())
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        n, T, models = _batch_spec(case)
        seeds = rng.integers(1, 1 << 31, len(n)).astype(np.uint32)
        s["batch"] = vc.FilterBatch(n, T, seeds, models,
                                    vc.SCHEMES[case["scheme"]], 0.5)
        s["obs"] = np.concatenate(
            [_simulate(rng, int(t), m) for t, m in zip(T, models)])
        s["hist"] = _histories(int(T.sum()))
    elif kind == "learned":
        rng = np.random.default_rng(seed)
        s["net"] = vc.Proposal(seed)
        s["net"].params.copy_(_gpu(np.concatenate(
            [w.ravel() for w in _network(rng)])))
        s["net"].pack()
        nf, T = case["nf"], case["T"]
        model = vc.bearings_model()
        s["batch"] = vc.FilterBatch(
            [case["n"]] * nf, [T] * nf, seed + 1 + np.arange(nf),
            [model] * nf, vc.SCHEMES[case["scheme"]], 0.5, bearings=True,
            packed=s["net"].packed.data_ptr())
        s["obs"] = np.tile(_simulate_bearings(rng, T, model), nf)
        s["hist"] = _histories(nf * T)
    elif kind == "resample":
        n = case["n"]
        s["W"] = torch.softmax(_log_weights(case, seed), 0)
        s["engine"] = vc.rng(vc.PHILOX4X32, seed + 1)
        s["rep"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        if case["select"]:
            s["idx"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            g = torch.Generator(device="cuda").manual_seed(seed + 2)
            s["state"] = torch.randn(4, n, device="cuda", generator=g)
    elif kind == "weight":
        n = case["n"]
        l = _log_weights(case, seed)
        s["in"] = torch.exp(l) if case["op"] == "set" else l
        s["W0"] = torch.softmax(_log_weights(case, seed + 1000), 0)
        s["W"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        s["ess"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(seed + 2)
        s["state"] = torch.randn(2, n, dtype=torch.float64, device="cuda",
                                 generator=g)
        s["mean"] = torch.zeros(2, dtype=torch.float64, device="cuda")
    elif kind == "rng":
        k = vc.PHILOX4X32 if case["engine"] == "philox" else vc.THREEFRY4X64
        s["engine"] = vc.rng(k, seed + 1)
        if case["dist"] == "rand":
            dt = torch.int32 if case["engine"] == "philox" else torch.int64
        else:
            dt = torch.float64 if case["bits"] == 64 else torch.float32
        s["out"] = torch.zeros(case["n"], dtype=dt, device="cuda")
    else:
        W, feat, nu = _mlp_inputs(case, seed)
        s["net"] = vc.Proposal(seed)
        s["net"].params.copy_(_gpu(np.concatenate([w.ravel() for w in W])))
        s["net"].pack()
        s["feat"], s["nu"] = _gpu(feat), _gpu(nu)
        s["loss"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        s["grad"] = torch.zeros(s["net"].nparams, device="cuda")
        s["out"] = torch.zeros(case["B"], 8, device="cuda")
    return s


# --------------------------------------------------------------------- run


def _engine_state(r):
    """The engine's position after a call (counter limbs, next word)."""
    return np.array([int(v) & 0x7FFFFFFFFFFFFFFF for v in r.ctr] + [r.index],
                    np.int64)


class _DeviceArray:
    """A device buffer of the library's, for torch; holds its owner (a
    tensor made from it holds this object)."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "data": (ptr, False), "shape": shape, "strides": strides,
            "typestr": typestr, "version": 3}


def _particles(pf):
    """The filter's particles (4 rows) and weights after a run."""
    e = pf.precision // 8
    ld = (pf.n + 255) // 256 * 256
    state, weight = pf.state_ptrs()
    return [torch.as_tensor(_DeviceArray(pf, p, shape, strides,
                                         "<f%d" % e), device="cuda")
            for p, shape, strides in ((state, (4, pf.n), (e * ld, e)),
                                      (weight, (pf.n,), None))]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pf":
        out = s["pf"].run(s["obs"])
        out["state"], out["weight"] = _particles(s["pf"])
        return out
    if kind in ("batch", "learned"):
        mean, ess, res, logz = s["hist"]
        vc.call("vsmc_cuda_batch_run", s["batch"].handle, s["obs"].ctypes.data,
                mean.ctypes.data, ess.ctypes.data, res.ctypes.data,
                logz.ctypes.data)
        return [mean, ess, res, logz]
    # a default stream of torch's is the legacy stream of the C ABI
    if kind == "resample":
        n = case["n"]
        r = vc.Rng.from_buffer_copy(s["engine"])
        vc.call("vsmc_cuda_resample", n, n, ctypes.byref(r),
                s["W"].data_ptr(), s["rep"].data_ptr(),
                vc.SCHEMES[case["scheme"]], None)
        out = [s["rep"], _engine_state(r)]
        if case["select"]:
            vc.call("vsmc_cuda_resample_trans_rep_index", n, n,
                    s["rep"].data_ptr(), s["idx"].data_ptr(), None)
            vc.call("vsmc_cuda_state_copy_f32", n, 4, s["idx"].data_ptr(),
                    s["state"].data_ptr(), None)
            out += [s["idx"], s["state"]]
        return out
    if kind == "weight":
        n, op = case["n"], case["op"]
        if op == "add_log":
            s["W"].copy_(s["W0"])
        vc.call("vsmc_cuda_weight_" + op, n, s["in"].data_ptr(),
                s["W"].data_ptr(), s["ess"].data_ptr(), None)
        vc.call("vsmc_cuda_monitor_mean_f64", n, 2, s["state"].data_ptr(),
                s["W"].data_ptr(), s["mean"].data_ptr(), None)
        return [s["W"], s["ess"], s["mean"]]
    if kind == "rng":
        n, dist = case["n"], case["dist"]
        f32 = "_f32" if case["bits"] == 32 else ""
        r = vc.Rng.from_buffer_copy(s["engine"])
        out = s["out"].data_ptr()
        if dist == "normal":
            vc.call("vsmc_cuda_rng_normal" + f32, ctypes.byref(r), n, out,
                    0.0, 1.0, None)
        elif dist == "student_t":
            vc.call("vsmc_cuda_rng_student_t", ctypes.byref(r), n, out, 10.0,
                    None)
        else:
            vc.call("vsmc_cuda_rng_" + dist + f32, ctypes.byref(r), n, out,
                    None)
        return [s["out"], _engine_state(r)]
    net, B = s["net"], case["B"]
    if case["op"] == "forward":
        vc.call("vsmc_cuda_mlp_forward", net.packed.data_ptr(), B,
                s["feat"].data_ptr(), s["out"].data_ptr(), None)
        return s["out"]
    vc.call("vsmc_cuda_mlp_loss_grad", net.packed.data_ptr(), B,
            s["feat"].data_ptr(), s["nu"].data_ptr(), s["loss"].data_ptr(),
            s["grad"].data_ptr(), None)
    return [s["loss"], s["grad"]]


def work(case):
    """Bytes and operations one pass cannot do without.  A filter step reads
    and writes every particle's state and weight; operations count a normal
    or a transcendental as one."""
    kind = case["kind"]
    if kind == "pf":
        e = case["precision"] // 8
        steps = case["n"] * case["T"]
        return {"bytes": 10 * e * steps, "flops": 60 * steps}
    if kind == "batch":
        mean_n = (case["nmax"] - case["nmin"]) / math.log(
            case["nmax"] / case["nmin"])
        steps = case["nf"] * mean_n * (case["Tmin"] + case["Tmax"]) / 2
        return {"bytes": 40 * steps, "flops": 60 * steps}
    if kind == "learned":
        steps = case["nf"] * case["n"] * case["T"]
        return {"bytes": 40 * steps,
                "flops": 2 * (6 * 64 + 64 * 64 + 64 * 8) * steps}
    if kind == "resample":
        n = case["n"]
        if case["select"]:  # weights, counts, parents, moved particles
            return {"bytes": (8 + 4 + 4 + 16) * n, "flops": 4 * n}
        return {"bytes": 12 * n, "flops": 4 * n}
    if kind == "weight":
        n = case["n"]
        return {"bytes": (8 + 8 + 16) * n, "flops": 10 * n}
    if kind == "rng":
        wide = case["bits"] == 64 and not (
            case["dist"] == "rand" and case["engine"] == "philox")
        return {"bytes": (8 if wide else 4) * case["n"],
                "flops": 20 * case["n"]}
    mac = 6 * 64 + 64 * 64 + 64 * 8
    B = case["B"]
    if case["op"] == "forward":
        return {"bytes": (24 + 32) * B, "flops": 2 * mac * B}
    return {"bytes": 40 * B, "flops": 6 * mac * B}


# ------------------------------------------------- the same in 64 bits


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 blocks (uint64 arrays holding 32-bit words)."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, np.uint64) for v in (c0, c1, c2, c3)]
    k0, k1 = int(k0), int(k1)
    sh = np.uint64(32)
    for r in range(10):
        if r:
            k0 = (k0 + 0x9E3779B9) & 0xFFFFFFFF
            k1 = (k1 + 0xBB67AE85) & 0xFFFFFFFF
        a = c[2] * np.uint64(0xCD9E8D57)
        b = c[0] * np.uint64(0xD2511F53)
        c = [(a >> sh) ^ np.uint64(k0) ^ c[1], a & m,
             (b >> sh) ^ np.uint64(k1) ^ c[3], b & m]
    return c


def _stream(seed, n):
    """The first n words of CounterEngine(seed), Philox4x32."""
    nb = (n + 3) // 4
    w = _philox(np.arange(1, nb + 1, dtype=np.uint64),
                *[np.zeros(nb, np.uint64)] * 3, seed, 0)
    return np.stack(w, 1).reshape(-1)[:n]


def _normal_batch(words, n):
    """The batch layout of normal_distribution from its uniforms' words."""
    u = words.astype(np.float64) * 2.0 ** -32
    out = np.empty(n)
    full = n // 1024 * 1024
    for lo, hi, k in ((0, full, 1024), (full, n, n - full)):
        nu = k // 2
        if hi > lo and nu:
            v = u[lo:lo + (hi - lo) // k * k].reshape(-1, k)
            r = np.sqrt(-2.0 * np.log(v[:, :nu]))
            th = 2 * np.pi * v[:, nu:2 * nu]
            out[lo:hi].reshape(-1, k)[:, :2 * nu] = np.concatenate(
                [r * np.sin(th), r * np.cos(th)], 1)
    if n % 2:
        out[n - 1] = math.sqrt(-2.0 * math.log(u[n])) * math.cos(
            2 * math.pi * u[n + 1])
    return out


def _normalized(w):
    W = w * (1.0 / np.cumsum(w)[-1])
    return W, 1.0 / np.cumsum(W * W)[-1]


def _exact_pf64(case, seed):
    """The bootstrap filter in numpy doubles (left-to-right sums)."""
    if case["scheme"] not in ("stratified", "systematic"):
        return None
    m = vc.default_model()
    n, T, strat = case["n"], case["T"], case["scheme"] == "stratified"
    obs = _simulate(np.random.default_rng(seed), T, m)
    key = seed + 1
    h = 0.5 * m.dt * m.dt
    c2 = 2 * (math.lgamma(0.5 * (m.nu + 1)) - math.lgamma(0.5 * m.nu) -
              0.5 * math.log(m.nu * math.pi) - math.log(m.obs_scale))
    i = np.arange(n, dtype=np.uint64)
    one, zero = np.ones(n, np.uint64), np.zeros(n, np.uint64)
    delta = 1.0 / n
    pos = 0  # words taken from the resampling engine
    W = np.full(n, 1.0 / n)
    logz = 0.0
    mean, ess, res, lz = _histories(T)

    def pair(a, b):
        r = np.sqrt(-2.0 * np.log(a * 2.0 ** -32))
        th = 2 * np.pi * (b * 2.0 ** -32)
        return r * np.cos(th), r * np.sin(th)

    for t in range(T):
        w = [v.astype(np.float64) for v in _philox(one, i, zero, zero, t, key)]
        if t == 0:
            z1, z2 = pair(w[0], w[1])
            z3, z4 = pair(w[2], w[3])
            S = np.stack([m.sd_pos0 * z1, m.sd_pos0 * z2, m.sd_vel0 * z3,
                          m.sd_vel0 * z4])
        else:
            a = np.stack(pair(w[0], w[1])) * m.sigma_a
            S = np.concatenate([S[:2] + m.dt * S[2:] + h * a,
                                S[2:] + m.dt * a])
        z = (obs[t][:, None] - S[:2]) / m.obs_scale
        ll = c2 - 0.5 * (m.nu + 1) * np.log1p(z * z / m.nu).sum(0)
        top = ll.max()
        logz += top + math.log((W * np.exp(ll - top)).sum())
        lw = ll if t == 0 else np.log(W) + ll
        W, e = _normalized(np.exp(lw - lw.max()))
        ess[t], lz[t] = e, logz
        if e < case["threshold"] * n:
            res[t] = 1
            nw = n if strat else 1
            b = np.arange(pos // 4, (pos + nw - 1) // 4 + 1, dtype=np.uint64)
            o = np.ones(len(b), np.uint64)
            wd = np.stack(_philox(b + np.uint64(1), 0 * o, o, 0 * o, 0, key),
                          1).reshape(-1)[pos % 4:][:nw]
            u = wd * 2.0 ** -32 * delta + np.arange(n) * delta
            F = np.searchsorted(np.maximum.accumulate(u),
                                np.cumsum(W[:-1]), side="right")
            rep = np.diff(np.concatenate([[0], F, [n]]))
            pos += min(n, n - int(rep[-1]) + 1) if strat else 1
            idx = np.where(rep > 0, np.arange(n), 0)
            idx[rep == 0] = np.repeat(np.arange(n), np.maximum(rep - 1, 0))
            S = S[:, idx]
            W, _ = _normalized(np.full(n, 1.0 / n))
        mean[t] = S[:2] @ W
    return {"mean": mean, "ess": ess, "resampled": None, "logz": lz,
            "state": S, "weight": W}


def _exact_mlp(case, seed):
    W, feat, nu = _mlp_inputs(case, seed)
    W = [torch.from_numpy(w).double().requires_grad_() for w in W]
    a = torch.from_numpy(feat).double()
    for k in (0, 2):
        a = torch.nn.functional.gelu(a @ W[k].T + W[k + 1],
                                     approximate="tanh")
    out = a @ W[4].T + W[5]
    if case["op"] == "forward":
        return out.detach()
    mu, l = out[:, :4], out[:, 4:]
    d = torch.from_numpy(nu).double() - mu
    loss = (0.5 * (d * d * torch.exp(-l) + l)).sum(1).mean()
    g = torch.autograd.grad(loss, W)
    return [loss.detach().reshape(1), torch.cat([x.reshape(-1) for x in g])]


def exact(case, seed):
    kind = case["kind"]
    if kind == "pf" and case["precision"] == 64:
        return _exact_pf64(case, seed)
    if kind == "weight":
        s = prepare(case, seed)
        l = s["in"].cpu().numpy()
        if case["op"] == "set":
            w = l
        else:
            if case["op"] == "add_log":
                l = np.log(s["W0"].cpu().numpy()) + l
            w = np.exp(l - l.max())
        W, ess = _normalized(w)
        return [W, np.array([ess]), s["state"].cpu().numpy() @ W]
    if kind == "rng" and case["engine"] == "philox":
        n = case["n"]
        if case["dist"] == "u01":
            w = _stream(seed + 1, n)
            if case["bits"] == 32:
                return [(w >> np.uint64(8)).astype(np.float64) * 2.0 ** -24,
                        None]
            return [w.astype(np.float64) * 2.0 ** -32, None]
        if case["dist"] == "normal":
            w = _stream(seed + 1, n + 2)
            if case["bits"] == 32:
                w = (w >> np.uint64(8)) << np.uint64(8)
            return [_normal_batch(w, n), None]
    if kind == "mlp":
        return _exact_mlp(case, seed)
    # replication counts, words and parents are whole numbers; a precision-32
    # filter's path hangs on its own rounded weights; Student-t variates and
    # the Threefry engine would need the library's own stream logic
    return None
