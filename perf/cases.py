"""Measured workloads of the extended-likelihood engine.

A case is one call that an analysis makes: an evaluation of the likelihood by
a minimiser, the Hessian at the end of a fit, a normalisation integral, the
decay amplitudes of an event sample, the batched evaluation and the batched
fit of many kinematic bins, and the training of the warm-start network.  All
inputs are synthetic and follow from a seed.
"""
import math

import numpy as np
import torch

from rootpwa_gb300 import ampIntegralMatrix, pwaLikelihood, pwaMLP, pwaMultibin
from rootpwa_gb300.isobar import isobarCanonicalAmplitudes, isobarHelicityAmplitudes

M_PI = 0.13957039
DEV = "cuda"


def listed():
    return [
        # a small first analysis: one minimiser call with host buffers, bound by launch and latency
        dict(name="fdf_15w_20k", kind="fdf", n_neg=0, n_pos=15, rank=1, events=20_000, entry="host", mixing=0),
        # the production likelihood of a three-pion wave set, parameters and result on the device
        dict(name="fdf_87w_1M", kind="fdf", n_neg=7, n_pos=80, rank=2, events=1_000_000, entry="device", mixing=8),
        # a rank-4 spin-density matrix, both reflectivities, a ragged number of events
        dict(name="fdf_64w_r4", kind="fdf", n_neg=10, n_pos=54, rank=4, events=200_003, entry="host", mixing=8),
        # error matrix after a production fit
        dict(name="hessian_87w", kind="hessian", n_neg=7, n_pos=80, rank=2, events=250_001, mixing=8),
        # normalisation integral of the production wave set, split-precision tensor-core path
        dict(name="integral_tf32x3_5M", kind="integral", waves=87, events=5_000_000, precision="tf32x3", weights=False,
             source="device", mixing=8),
        # importance-sampled Monte Carlo of a mass bin with the default precision
        dict(name="integral_fp32", kind="integral", waves=50, events=300_001, precision="fp32", weights=True,
             source="device", mixing=0),
        # the reference's own precision, as used to check an analysis
        dict(name="integral_fp64", kind="integral", waves=87, events=150_000, precision="fp64", weights=False,
             source="device", mixing=8),
        # decay amplitudes of a data sample into the likelihood's single-precision store
        dict(name="isobar_c64", kind="isobar", waves=88, events=300_000, dtype="complex64", formalism="helicity"),
        # the same in double precision, for a smaller sample
        dict(name="isobar_c128", kind="isobar", waves=88, events=40_001, dtype="complex128", formalism="helicity"),
        # one evaluation of every bin and start point of a mass-binned fit (64 starts)
        dict(name="multibin_fdf_64", kind="multibin_fdf", bins=24, waves=50, starts=64, median=40_000, group=32),
        # a whole multi-start fit of a few bins
        dict(name="multibin_fit", kind="multibin_fit", bins=8, waves=50, starts=64, median=40_000, group=32),
        # training of the warm-start network: 256-row steps of the 5203-512-512-102 perceptron
        dict(name="mlp_train", kind="mlp_train", n_in=5203, hidden=512, n_out=102, rows=2048, batch=256, epochs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fdf", "fdf", "fdf", "hessian", "integral", "integral", "isobar", "isobar", "multibin_fdf",
                       "multibin_fit", "mlp_train"])
    if kind in ("fdf", "hessian"):
        rank = rng.randint(1, 4)
        top = {1: 140, 2: 110, 3: 80, 4: 64}[rank] if kind == "fdf" else {1: 110, 2: 88, 3: 50, 4: 40}[rank]
        n = max(rank, _log_int(rng, 4, top))
        n_neg = rng.choice([0, 0, max(1, n // 10), n // 4])
        c = dict(kind=kind, n_neg=n_neg, n_pos=n - n_neg, rank=rank,
                 events=_log_int(rng, 2_000, 1_000_000 if kind == "fdf" else 250_000), mixing=rng.choice([0, 8]))
        if kind == "fdf":
            c["entry"] = rng.choice(["host", "host", "device", "value"])
        return c
    if kind == "integral":
        precision = rng.choice(["fp32", "tf32x3", "bf16x3", "fp64"])
        return dict(kind=kind, waves=_log_int(rng, 5, 120), precision=precision,
                    events=_log_int(rng, 5_000, 100_000 if precision == "fp64" else 1_000_000),
                    weights=rng.random() < 0.4, source=rng.choice(["device", "device", "host"]),
                    mixing=rng.choice([0, 8]))
    if kind == "isobar":
        dtype = rng.choice(["complex64", "complex128"])
        return dict(kind=kind, waves=_log_int(rng, 6, 88),
                    events=_log_int(rng, 500, 300_000 if dtype == "complex64" else 40_000), dtype=dtype,
                    formalism=rng.choice(["helicity", "helicity", "canonical"]))
    if kind == "multibin_fdf":
        group = rng.choice([8, 32])
        return dict(kind=kind, bins=rng.randint(1, 24), waves=rng.randint(8, 60),
                    starts=rng.randint(1, 8) if group == 8 else rng.randint(9, 64),
                    median=_log_int(rng, 3_000, 40_000), group=group)
    if kind == "multibin_fit":
        group = rng.choice([8, 32])
        return dict(kind=kind, bins=rng.randint(1, 8), waves=rng.randint(8, 50),
                    starts=5 if group == 8 else rng.randint(9, 64), median=_log_int(rng, 3_000, 40_000), group=group)
    w = rng.randint(10, 50) + 1
    return dict(kind=kind, n_in=2 * w * w + 1, hidden=512, n_out=2 * w, rows=rng.choice([512, 1000, 2048]),
                batch=rng.choice([64, 128, 256]), epochs=rng.randint(1, 3))


# -- inputs -------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _cn(g, *shape):
    """complex64 draws with re, im ~ N(0, 1)."""
    return torch.complex(torch.randn(*shape, generator=g, device=DEV), torch.randn(*shape, generator=g, device=DEV))


def _sigma(seed, n_waves):
    """wave scales, log-uniform over two decades."""
    r = np.random.default_rng([int(seed) % (1 << 62), 1])
    return torch.from_numpy(np.exp(r.uniform(math.log(0.1), math.log(10.0), n_waves)).astype(np.float32)).to(DEV)


def _amps(g, sigma, n, mixing):
    """complex64 [wave][event]: independent waves, or waves that share `mixing` complex sources."""
    W = len(sigma)
    z = _cn(g, W, n)
    if mixing:
        B = _cn(g, W, mixing) / math.sqrt(2.0 * mixing)
        c = _cn(g, mixing, n)
        for w in range(W):
            z[w] += (B[w, :, None] * c).sum(dim=0)
        z *= math.sqrt(0.5)
    z *= sigma[:, None]
    return z.contiguous()


def _gram(a, weights=None, chunk=1 << 16):
    """sum_k w_k a_ik conj(a_jk) in complex128."""
    out = torch.zeros(a.shape[0], a.shape[0], dtype=torch.complex128, device=a.device)
    for b in range(0, a.shape[1], chunk):
        x = a[:, b:b + chunk].to(torch.complex128)
        y = x if weights is None else x * weights[None, b:b + chunk]
        out += y @ x.conj().T
    return out


def _integrals(g, sigma, mixing, n_mc):
    """raw normalisation and acceptance sums of a Monte Carlo sample and their event counts."""
    mc = _amps(g, sigma, n_mc, mixing)
    acc = torch.rand(n_mc, generator=g, device=DEV) < 0.6
    n_acc = int(acc.sum())
    return _gram(mc).cpu().numpy(), _gram(mc[:, acc]).cpu().numpy(), n_mc, n_acc


def _integral_object(names, sums, events):
    I = ampIntegralMatrix()
    I.setWaveNames(names)
    I.setMatrix(sums)
    I.setNmbEvents(events)
    return I


def _names(n_neg, n_pos):
    return (["n%03d" % i for i in range(n_neg)] + ["p%03d" % i for i in range(n_pos)],
            [-1] * n_neg + [+1] * n_pos)


def _likelihood(names, refl, rank, data, ints):
    L = pwaLikelihood()
    L.init(names, refl, None, rank, 0.0)
    L.addNormIntegral(_integral_object(names, ints[0], ints[2]))
    L.addAccIntegral(_integral_object(names, ints[1], ints[3]))
    for k, n in enumerate(names):
        L.addAmplitude(n, data[k])
    # no timing of kernel variants: which of them wins may depend on the moment, and with it the last bits of the
    # results; an analysis that is to give the same numbers in every process turns it off
    L.setAutotune(False)
    L.finishInit()
    return L


def _slots(n_neg, n_pos, rank):
    """parameter index of (re, im) of each production amplitude [rank][wave], -1 where there is none:
    amplitude w of a reflectivity exists from rank index <= w on and is real where they are equal."""
    W = n_neg + n_pos
    re, im = -np.ones((rank, W), dtype=np.int64), -np.ones((rank, W), dtype=np.int64)
    p = 0
    for r in range(rank):
        for off, n in ((0, n_neg), (n_neg, n_pos)):
            for w in range(r, n):
                re[r, off + w] = p
                p += 1
                if w > r:
                    im[r, off + w] = p
                    p += 1
    return re, im, p + 1


def _fdf_inputs(case, seed):
    W = case["n_neg"] + case["n_pos"]
    g = _gen(seed)
    sigma = _sigma(seed, W)
    data = _amps(g, sigma, case["events"], case["mixing"])
    ints = _integrals(g, sigma, case["mixing"], 20 * W + 4000)
    P = _slots(case["n_neg"], case["n_pos"], case["rank"])[2]
    par = np.random.default_rng([int(seed) % (1 << 62), 2]).standard_normal(P)
    return data, ints, par


def _bins_inputs(case, seed):
    """per bin: data drawn in proportion to |V A|^2 + flat^2 of production amplitudes of its own, integrals."""
    W = case["waves"]
    r = np.random.default_rng([int(seed) % (1 << 62), 3])
    sizes = np.random.default_rng([case["bins"], case["median"]])  # the same event counts for every seed
    bins = []
    for b in range(case["bins"]):
        n = int(min(max(case["median"] * math.exp(sizes.normal(0.0, 1.0)), case["median"] / 20), case["median"] * 4))
        g = _gen(seed * 1000003 + b)
        sigma = _sigma(seed * 31 + b, W)
        v = torch.from_numpy((r.standard_normal(W) + 1j * r.standard_normal(W)).astype(np.complex64)).to(DEV)
        flat = abs(r.standard_normal())
        u = v.conj() * sigma                       # V A = sum conj(u) z with A = sigma z
        norm = float(u.abs().square().sum().sqrt())
        u = u / norm
        z = _cn(g, W, n)
        along = (u.conj()[:, None] * z).sum(dim=0)
        # |along|^2 / 2 ~ Exp(1), weighted by 2 norm^2 x + flat^2: a mixture of Gamma(2) and Exp(1)
        x = -torch.log1p(-torch.rand(n, generator=g, device=DEV))
        y = -torch.log1p(-torch.rand(n, generator=g, device=DEV))
        more = torch.rand(n, generator=g, device=DEV) < 2 * norm * norm / (2 * norm * norm + flat * flat)
        want = torch.sqrt(2.0 * (x + torch.where(more, y, torch.zeros_like(y))))
        z += u[:, None] * (along * (want / along.abs().clamp_min(1e-20)) - along)
        bins.append(((z * sigma[:, None]).contiguous(), _integrals(g, sigma, 0, 40 * W + 2000)))
    Q, P = case["bins"] * case["starts"], 2 * W  # 2 W - 1 amplitude components and the flat wave
    return bins, r.standard_normal((Q, P))


def _three_body(case, seed):
    """lab momenta of beam (N, 3) and final state (3, N, 3) of X -> pi- pi+ pi- at 190 GeV/c."""
    n, g = case["events"], _gen(seed)

    def uni(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)

    def direction():
        c, p = uni(-1, 1), uni(0, 2 * math.pi)
        s = torch.sqrt(1 - c * c)
        return torch.stack([s * torch.cos(p), s * torch.sin(p), c], dim=1)

    def boost(p, e, b):
        ga = 1 / torch.sqrt(1 - (b * b).sum(1))
        bp = (b * p).sum(1)
        k = ga * ga / (ga + 1) * bp + ga * e
        return p + k[:, None] * b, ga * (e + bp)

    def q2(M, a, b):
        return (M * M - (a + b) ** 2) * (M * M - (a - b) ** 2) / (4 * M * M)

    beam = torch.stack([0.05 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64),
                        0.05 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64),
                        torch.full((n,), 190.0, dtype=torch.float64, device=DEV)], dim=1)
    MX = uni(0.9, 2.2)
    pX = beam * uni(0.95, 1.0)[:, None]
    pX[:, :2] += 0.3 * torch.randn(n, 2, generator=g, device=DEV, dtype=torch.float64)
    EX = torch.sqrt(MX * MX + (pX * pX).sum(1))
    m12 = torch.sqrt(uni(0, 1) * ((MX - M_PI) ** 2 - 4 * M_PI ** 2) * 0.9998 + 4 * M_PI ** 2 * 1.0001)
    k = torch.sqrt(q2(MX, m12, M_PI))[:, None] * direction()
    kk = torch.sqrt(q2(m12, M_PI, M_PI))[:, None] * direction()
    e12 = torch.sqrt(m12 * m12 + (k * k).sum(1))
    e1 = torch.sqrt(M_PI ** 2 + (kk * kk).sum(1))
    bI, bX = k / e12[:, None], pX / EX[:, None]
    out = [boost(-k, torch.sqrt(M_PI ** 2 + (k * k).sum(1)), bX)[0]]
    for sign in (1.0, -1.0):
        p, e = boost(sign * kk, e1, bI)
        out.append(boost(p, e, bX)[0])
    fs = torch.stack(out)
    return beam.contiguous(), fs.contiguous()


# isobars (2J, mass, width); no mass: the pi pi S-wave with fixed parameters
_ISOBARS = [(0, 0.0, 0.0), (2, 0.7690, 0.1509), (0, 0.980, 0.070), (4, 1.2751, 0.1851), (0, 1.505, 0.109),
            (6, 1.6888, 0.161)]


def _waves(n):
    """pi- pi+ pi- waves (spins doubled), J <= 3, M <= 2, L <= 4, parity conserving, one in ten of negative
    reflectivity: (J, P, M, refl, L, isobar)."""
    def of(refl):
        out = []
        for J in (0, 2, 4, 6):
            for P in (-1, 1):
                for M in range(0, min(J, 4) + 1, 2):
                    if M == 0 and refl * P * (-1) ** (J // 2) == 1:
                        continue
                    for k, (j, _, _) in enumerate(_ISOBARS):
                        for L in range(0, 9, 2):
                            if (-1) ** (L // 2 + j // 2 + 1) == P and abs(L - j) <= J <= L + j:
                                out.append((J, P, M, refl, L, k))
        return out
    n_neg = n // 11
    return of(+1)[:n - n_neg] + of(-1)[:n_neg]


def _isobar_object(case):
    amp = (isobarCanonicalAmplitudes if case["formalism"] == "canonical" else isobarHelicityAmplitudes)()
    amp.setFinalState(["pi-", "pi+", "pi-"], [M_PI] * 3, beamMass=M_PI)
    for J, P, M, refl, L, k in _waves(case["waves"]):
        j, mass, width = _ISOBARS[k]
        amp.addWave(J=J, P=P, M=M, refl=refl, L=L, S=j, isobarJ=j, isobarL=j,
                    massDependence="relativisticBreitWigner" if mass else "piPiSWaveAuMorganPenningtonKachaev",
                    isobarMass=mass, isobarWidth=width, isobarDaughters=(1, 2), bachelor=0, isobarName="iso%d" % k)
    return amp


def _mc_weights(case, seed):
    if not case["weights"]:
        return None
    return np.random.default_rng([int(seed) % (1 << 62), 4]).uniform(0.2, 2.0, case["events"])


def _mlp_inputs(case, seed):
    r = np.random.default_rng([int(seed) % (1 << 62), 5])
    X = r.standard_normal((case["rows"], case["n_in"]), dtype=np.float32)
    T = (0.1 * r.standard_normal((case["rows"], case["n_out"]), dtype=np.float32)).astype(np.float32)
    return X, T


# -- the calls ----------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("fdf", "hessian"):
        data, ints, par = _fdf_inputs(case, seed)
        names, refl = _names(case["n_neg"], case["n_pos"])
        s["L"] = _likelihood(names, refl, case["rank"], data, ints)
        s["par"] = par
        if case.get("entry") == "device":
            s["d_par"] = torch.from_numpy(par).to(DEV)
            s["d_out"] = torch.zeros(len(par) + 2, dtype=torch.float64, device=DEV)
            s["stream"] = torch.cuda.Stream()
    elif kind == "integral":
        s["names"] = ["w%03d" % i for i in range(case["waves"])]
        a = _amps(_gen(seed), _sigma(seed, case["waves"]), case["events"], case["mixing"])
        s["amps"] = a if case["source"] == "device" else a.cpu().numpy()
        s["weights"] = _mc_weights(case, seed)
        s["I"] = ampIntegralMatrix()
    elif kind == "isobar":
        s["amp"] = _isobar_object(case)
        s["beam"], s["fs"] = _three_body(case, seed)
    elif kind in ("multibin_fdf", "multibin_fit"):
        bins, s["x"] = _bins_inputs(case, seed)
        names, refl = _names(0, case["waves"])
        s["M"] = pwaMultibin()
        s["M"].setOptions(startGroup=case["group"])
        for data, ints in bins:
            s["M"].addBin(_likelihood(names, refl, 1, data, ints), case["starts"])
    else:
        s["X"], s["T"] = _mlp_inputs(case, seed)
        s["net"] = pwaMLP(case["n_in"], case["hidden"], case["hidden"], case["n_out"], seed=int(seed) % 1000)
        s["p0"] = s["net"].params()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fdf":
        if case["entry"] == "device":
            s["L"].FdFDevice(s["d_par"].data_ptr(), s["d_out"].data_ptr(), stream=s["stream"].cuda_stream)
            return s["d_out"]
        if case["entry"] == "value":
            return s["L"].DoEval(s["par"])
        f, g = s["L"].FdF(s["par"])
        return {"f": f, "g": g}
    if kind == "hessian":
        return s["L"].Hessian(s["par"])
    if kind == "integral":
        s["I"].integrate(s["names"], s["amps"], weights=s["weights"], precision=case["precision"])
        return {"sums": s["I"].matrix(), "events": s["I"].nmbEvents()}
    if kind == "isobar":
        return s["amp"].amplitudes(s["beam"], s["fs"], dtype=case["dtype"])
    if kind == "multibin_fdf":
        f, g = s["M"].FdF(s["x"])
        return {"f": f, "g": g}
    if kind == "multibin_fit":
        r = s["M"].fit(s["x"])
        return {k: r[k] for k in ("x", "f", "gnorm", "status", "iterations")}
    s["net"].setParams(s["p0"])
    history = s["net"].train(s["X"], s["T"], batch=case["batch"], epochs=case["epochs"])
    return {"history": history, "params": s["net"].params()}


def work(case):
    kind = case["kind"]
    if kind == "fdf":
        W, n, r = case["n_neg"] + case["n_pos"], case["events"], case["rank"]
        return {"bytes": 8 * W * n, "flops": (1 if case["entry"] == "value" else 2) * 8 * W * r * n}
    if kind == "hessian":
        W, n, r = case["n_neg"] + case["n_pos"], case["events"], case["rank"]
        s = r * W
        # the products d d^H and d d^T of the rank x wave slots (each symmetric) and A A^H
        return {"bytes": 8 * W * n, "flops": 8 * n * (s * (s + 1) + W * (W + 1) // 2)}
    if kind == "integral":
        W, n = case["waves"], case["events"]
        return {"bytes": 8 * W * n + 16 * W * W, "flops": 8 * n * W * (W + 1) // 2}
    if kind == "isobar":
        W, n = case["waves"], case["events"]
        size = 8 if case["dtype"] == "complex64" else 16
        # per wave and Bose term: the D functions of both vertices, barrier factors and the Breit-Wigner
        return {"bytes": n * (96 + size * W), "flops": n * W * 2 * 100}
    if kind in ("multibin_fdf", "multibin_fit"):
        sizes = np.random.default_rng([case["bins"], case["median"]])
        n = sum(int(min(max(case["median"] * math.exp(sizes.normal(0.0, 1.0)), case["median"] / 20),
                        case["median"] * 4)) for _ in range(case["bins"]))
        # a fit evaluates a start point some fifty times
        times = 1 if kind == "multibin_fdf" else 50
        return {"bytes": times * 8 * case["waves"] * n, "flops": times * 16 * case["waves"] * case["starts"] * n}
    weights = case["n_in"] * case["hidden"] + case["hidden"] ** 2 + case["hidden"] * case["n_out"]
    steps = case["epochs"] * (case["rows"] // case["batch"])
    return {"bytes": 4 * case["rows"] * (case["n_in"] + case["n_out"]) + 8 * weights + steps * 28 * weights,
            "flops": 6 * weights * case["batch"] * steps}


# -- the same in 64 bits ------------------------------------------------------------

def _normalised(ints):
    """amplitude divisors, acceptance matrix per event in the normalised amplitudes, total acceptance."""
    norm, acc, n_norm, n_acc = ints
    d = np.sqrt(np.real(np.diag(norm)) / n_norm)
    return (torch.from_numpy(d).to(DEV), torch.from_numpy(acc / n_norm / np.outer(d, d)).to(DEV), n_acc / n_norm)


def _exact_fdf(case, data, ints, par):
    re, im, P = _slots(case["n_neg"], case["n_pos"], case["rank"])
    div, acc, tot = _normalised(ints)
    W, R, n0 = case["n_neg"] + case["n_pos"], case["rank"], case["n_neg"]
    V = torch.from_numpy(np.where(re >= 0, par[re], 0.0) + 1j * np.where(im >= 0, par[im], 0.0)).to(DEV)
    flat = par[-1]
    parts = [slice(0, n0), slice(n0, W)]
    f = 0.0
    G = torch.zeros(R, W, dtype=torch.complex128, device=DEV)
    c_sum = 0.0
    for b in range(0, data.shape[1], 1 << 16):
        A = data[:, b:b + (1 << 16)].to(torch.complex128) / div[:, None]
        S = [V[:, p] @ A[p] for p in parts]
        L = sum(x.abs().square().sum(0) for x in S) + flat * flat
        c = -2.0 / L
        f -= float(torch.log(L).sum())
        c_sum += float(c.sum())
        for p, x in zip(parts, S):
            G[:, p] += (c * x) @ A[p].conj().T
    for p in parts:
        D = V[:, p] @ acc[p, p].conj().T          # D_i = sum_j V_j conj(I_ij)
        f += float((V[:, p] * D.conj()).real.sum())
        G[:, p] += 2.0 * D
    f += flat * flat * tot
    g = np.zeros(P)
    Gh = G.cpu().numpy()
    g[re[re >= 0]] = Gh.real[re >= 0]
    g[im[im >= 0]] = Gh.imag[im >= 0]
    g[-1] = flat * c_sum + 2.0 * flat * tot
    return f, g


def _exact_hessian(case, data, ints, par):
    re, im, P = _slots(case["n_neg"], case["n_pos"], case["rank"])
    div, acc, tot = _normalised(ints)
    W, R, n0 = case["n_neg"] + case["n_pos"], case["rank"], case["n_neg"]
    V = torch.from_numpy(np.where(re >= 0, par[re], 0.0) + 1j * np.where(im >= 0, par[im], 0.0)).to(DEV)
    flat = par[-1]
    parts = [slice(0, n0), slice(n0, W)]
    row_re, row_im = torch.from_numpy(re.ravel()).to(DEV), torch.from_numpy(im.ravel()).to(DEV)
    H = torch.zeros(P, P, dtype=torch.float64, device=DEV)
    Gm = torch.zeros(W, W, dtype=torch.complex128, device=DEV)   # sum (2 / L) A_i conj(A_j)
    inv = 0.0
    for b in range(0, data.shape[1], 1 << 15):
        A = data[:, b:b + (1 << 15)].to(torch.complex128) / div[:, None]
        S = [V[:, p] @ A[p] for p in parts]
        L = sum(x.abs().square().sum(0) for x in S) + flat * flat
        d = torch.cat([x[:, None, :] * A[None, p].conj() for p, x in zip(parts, S)], dim=1).reshape(R * W, -1)
        J = torch.zeros(P, A.shape[1], dtype=torch.float64, device=DEV)
        J[row_re[row_re >= 0]] = d.real[row_re >= 0]
        J[row_im[row_im >= 0]] = d.imag[row_im >= 0]
        J[-1] = flat
        J *= 2.0 / L
        H += J @ J.T
        Gm += (A * (2.0 / L)) @ A.conj().T
        inv += float((2.0 / L).sum())
    B = 2.0 * acc - Gm
    full = torch.zeros_like(B)
    for p in parts:
        full[p, p] = B[p, p]
    Bh, out = full.cpu().numpy(), H.cpu().numpy()
    for r in range(R):
        k, l = re[r], im[r]
        ok, ol = k >= 0, l >= 0
        out[np.ix_(k[ok], k[ok])] += Bh.real[np.ix_(ok, ok)]
        out[np.ix_(k[ok], l[ol])] += Bh.imag[np.ix_(ok, ol)]
        out[np.ix_(l[ol], k[ok])] += Bh.imag[np.ix_(ok, ol)].T
        out[np.ix_(l[ol], l[ol])] += Bh.real[np.ix_(ol, ol)]
    out[-1, -1] += 2.0 * tot - inv
    return out


def _clebsch(j1, m1, j2, m2, J, M):
    """(j1 m1 j2 m2 | J M), arguments doubled (Racah)."""
    if (m1 + m2 != M or abs(m1) > j1 or abs(m2) > j2 or abs(M) > J or not abs(j1 - j2) <= J <= j1 + j2
            or (j1 + j2 + J) % 2 or (j1 + m1) % 2 or (j2 + m2) % 2):
        return 0.0

    def f(x):
        return math.factorial(x // 2)
    pre = ((J + 1) * f(J + j1 - j2) * f(J - j1 + j2) * f(j1 + j2 - J) / f(j1 + j2 + J + 2)
           * f(J + M) * f(J - M) * f(j1 - m1) * f(j1 + m1) * f(j2 - m2) * f(j2 + m2))
    s = 0.0
    for k in range(0, j1 + j2 + J + 1, 2):
        den = [k, j1 + j2 - J - k, j1 - m1 - k, j2 + m2 - k, J - j2 + m1 + k, J - j1 - m2 + k]
        if min(den) >= 0:
            s += (-1) ** (k // 2) / math.prod(f(x) for x in den)
    return math.sqrt(pre) * s


def _small_d(j, m, n, th):
    """Wigner's d^j_{m n}(theta), arguments doubled."""
    c, s = torch.cos(th / 2), torch.sin(th / 2)
    a, b, e, g = (j + m) // 2, (j - m) // 2, (j + n) // 2, (j - n) // 2
    root = math.sqrt(math.factorial(a) * math.factorial(b) * math.factorial(e) * math.factorial(g))
    out = torch.zeros_like(th)
    for k in range(max(0, (n - m) // 2), min(e, b) + 1):
        den = math.factorial(e - k) * math.factorial(k) * math.factorial((m - n) // 2 + k) * math.factorial(b - k)
        out += ((-1) ** ((m - n) // 2 + k) * root / den) * c ** (e + b - 2 * k) * s ** ((m - n) // 2 + 2 * k)
    return out


# |h_l|^2 z^(l + 1) of the spherical Hankel functions as polynomials in z = (q / 0.1973 GeV)^2
_HANKEL = [[1], [1, 1], [9, 3, 1], [225, 45, 6, 1], [11025, 1575, 135, 10, 1]]


def _barrier2(l, q):
    z = (q / 0.1973) ** 2
    poly = _HANKEL[l]
    return sum(poly) * z ** l / sum(k * z ** i for i, k in enumerate(poly))


def _q_squared(M, m):
    return (M * M - 4 * m * m) / 4


def _pipi_s(m):
    """pi pi S-wave, Au-Morgan-Pennington M solution in Kachaev's reduction (charged and neutral thresholds)."""
    mk = 0.5 * (0.493677 + 0.497611)
    s = m * m
    x = s / (4 * mk * mk) - 1
    K = 0.1131 / (s + 0.0074) + 0.0337 - 0.3185 * x - 0.0942 * x ** 2 - 0.5927 * x ** 3
    rho = 0
    for mp in (M_PI, 0.1349768):
        q2 = _q_squared(m, mp).to(torch.complex128)
        rho = rho + torch.sqrt(q2) / m
    return 1.0 / (K - 1j * rho)


def _exact_isobar(case, beam, fs):
    out = torch.zeros(case["waves"], case["events"], dtype=torch.complex128, device=DEV)

    def norm(p):
        return torch.sqrt((p * p).sum(1))

    def rest(p, e, P, E, M):
        e1 = (e * E - (p * P).sum(1)) / M
        return p - P * ((e + e1) / (E + M))[:, None], e1

    energy = [torch.sqrt(M_PI ** 2 + (p * p).sum(1)) for p in fs]
    pX, eX = fs[0] + fs[1] + fs[2], energy[0] + energy[1] + energy[2]
    nX = norm(pX)
    mX = torch.sqrt((eX - nX) * (eX + nX))
    z = rest(beam, torch.sqrt(M_PI ** 2 + (beam * beam).sum(1)), pX, eX, mX)[0]
    z = z / norm(z)[:, None]
    y = torch.linalg.cross(beam, pX)
    y = y / norm(y)[:, None]
    axes = [torch.linalg.cross(y, z), y, z]
    gj = []
    for p, e in zip(fs, energy):
        p1, e1 = rest(p, e, pX, eX, mX)
        gj.append((torch.stack([(p1 * a).sum(1) for a in axes], dim=1), e1))
    canonical = case["formalism"] == "canonical"
    for bach, a, b in ((0, 1, 2), (2, 1, 0)):      # the two pi- exchanged
        p, e = gj[a][0] + gj[b][0], gj[a][1] + gj[b][1]
        q = norm(p)
        m = torch.sqrt((e - q) * (e + q))
        if canonical:
            h = rest(gj[a][0], gj[a][1], p, e, m)[0]
        else:
            zh = p / q[:, None]
            yh = torch.stack([-p[:, 1], p[:, 0], torch.zeros_like(q)], dim=1)
            yh = yh / norm(yh)[:, None]
            xh = torch.linalg.cross(yh, zh)
            h = torch.stack([(gj[a][0] * xh).sum(1), (gj[a][0] * yh).sum(1),
                             (e * (gj[a][0] * zh).sum(1) - q * gj[a][1]) / m], dim=1)
        phi, theta = torch.atan2(p[:, 1], p[:, 0]), torch.atan2(torch.hypot(p[:, 0], p[:, 1]), p[:, 2])
        phh, thh = torch.atan2(h[:, 1], h[:, 0]), torch.atan2(torch.hypot(h[:, 0], h[:, 1]), h[:, 2])
        qh = norm(h)
        for w, (J, P, M, refl, L, k) in enumerate(_waves(case["waves"])):
            j, mass, width = _ISOBARS[k]
            if mass:
                q0 = math.sqrt(_q_squared(mass, M_PI))
                qm = torch.sqrt(_q_squared(m, M_PI).clamp_min(0))
                gamma = width * (mass / m) * (qm / q0) * (_barrier2(j // 2, qm) / _barrier2(j // 2, q0))
                bw = mass * width / (mass * mass - m * m - 1j * mass * gamma)
            else:
                bw = _pipi_s(m)
            f = refl * P * (-1) ** ((J - M) // 2)
            total = 0
            for lam in range(-j, j + 1, 2):
                if not canonical and abs(lam) > J:
                    continue
                own = torch.exp(0.5j * lam * phh) * _small_d(j, lam, 0, thh)

                def vertex(proj):
                    if canonical:
                        cg = _clebsch(L, proj - lam, j, lam, J, proj)
                        if cg == 0 or abs(proj - lam) > L:
                            return 0
                        return cg * torch.exp(0.5j * (proj - lam) * phi) * _small_d(L, proj - lam, 0, theta)
                    return torch.exp(0.5j * proj * phi) * _small_d(J, proj, lam, theta)
                x = vertex(M) if M == 0 else (vertex(M) - f * vertex(-M)) / math.sqrt(2.0)
                cg = 1.0 if canonical else _clebsch(L, 0, j, lam, J, lam)
                total = total + cg * x * own
            total = total * math.sqrt(L + 1) * math.sqrt(j + 1)
            out[w] += total * bw * torch.sqrt(_barrier2(L // 2, q) * _barrier2(j // 2, qh)) * math.sqrt(0.5)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fdf", "hessian"):
        data, ints, par = _fdf_inputs(case, seed)
        if kind == "hessian":
            return _exact_hessian(case, data, ints, par)
        f, g = _exact_fdf(case, data, ints, par)
        if case["entry"] == "device":
            return torch.from_numpy(np.concatenate([[f], g, [0.0]]))
        return f if case["entry"] == "value" else {"f": f, "g": g}
    if kind == "integral":
        a = _amps(_gen(seed), _sigma(seed, case["waves"]), case["events"], case["mixing"])
        w = _mc_weights(case, seed)
        if w is None:
            return {"sums": _gram(a).cpu().numpy(), "events": case["events"]}
        inv = torch.from_numpy(1.0 / w).to(DEV)
        return {"sums": (_gram(a, inv) * (case["events"] / inv.sum())).cpu().numpy(), "events": case["events"]}
    if kind == "isobar":
        return _exact_isobar(case, *_three_body(case, seed))
    if kind == "multibin_fdf":
        bins, x = _bins_inputs(case, seed)
        one = dict(n_neg=0, n_pos=case["waves"], rank=1)
        f, g = np.zeros(len(x)), np.zeros_like(x)
        for b, (data, ints) in enumerate(bins):
            for q in range(b * case["starts"], (b + 1) * case["starts"]):
                f[q], g[q] = _exact_fdf(one, data, ints, x[q])
        return {"f": f, "g": g}
    return None  # a whole fit and a whole training run: minutes in 64 bits
