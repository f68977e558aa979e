"""The measured cases of the LMM swaption-portfolio engine: what a user has it do, through its Python binding.

A case names a call, a model and a size. The calls are value and all Greeks in FP32 (device normals, host normals, in-kernel
Philox normals), the forward/backward pair an autograd node uses, the FP64 adjoint, the FP64 bump-and-revalue run, the
reference's own entry point, and the MRG32k3a normal stream. The FP32 calls deliver FP32-accurate sums in FP64 buffers; the
program here keeps them as FP32 tensors, as a PyTorch program that asked for FP32 Greeks does.
"""
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("financial-services-workload-samples_gb300")
C = P.configs

BUMP = 1e-6               # the bump of the headline workload's finite-difference check


def listed():
    return [
        # a desk's intraday revaluation of one portfolio: few paths, an odd number of them, latency counts
        dict(name="f32_3001", call="f32", model="flat", paths=3001),
        # the reference program's own run: its parameters, its 131,072 paths, FP32 build
        dict(name="f32_131072", call="f32", model="reference", paths=131072),
        # the headline workload end to end: normals in pinned host memory, results back on the host
        dict(name="f32_host_4194304", call="f32_host", model="flat", paths=4194304),
        # throughput mode: vol vector, normals generated in the kernel
        dict(name="philox_16777216", call="philox", model="volvec", paths=16777216),
        # scenario sweep: every curve on the same normals, one launch
        dict(name="curves_256x16384", call="f32", model="curves", curves=256, paths=16384),
        # long tenor: 160 rates, 120 steps, 30 swaptions, rates saved every 8 steps
        dict(name="long_1048576", call="f32", model="long", paths=1048576),
        # a shape of the user's own: 96 rates, 60 steps, random curve and vols, an odd path count
        dict(name="shape96x60_50001", call="f32", model="random", nn=96, nmat=60, nopt=8, paths=50001),
        # one step of a calibration through autograd: forward with a tape, then backward; a ragged path count
        dict(name="pair_300001", call="pair", model="volvec", paths=300001),
        # the reference method in FP64: its 65,536 paths
        dict(name="f64_65536", call="f64", model="flat", paths=65536),
        # plain FP64 forward with every input bumped, the method that the adjoint is measured against
        dict(name="bump_16384", call="bump", model="flat", paths=16384),
        # the reference's entry point called from a program like its main(): FP64, normals of its generator family, host array
        dict(name="entry_f64_131072", call="entry", model="reference", dtype="f64", paths=131072),
        # the generator alone, FP64, for the headline workload's normals
        dict(name="mrg_f64_167772160", call="mrg", dtype="f64", paths=4194304),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, even in its logarithm, most often odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v | 1 if rng.random() < 0.7 else v))


def draw(rng):
    call = rng.choice(["f32", "f32", "f32", "f32_host", "philox", "curves", "long", "shape", "pair", "f64", "bump", "entry", "mrg"])
    if call == "f32":
        return dict(call="f32", model=rng.choice(["flat", "reference", "volvec"]), paths=_log(rng, 1000, 4194304))
    if call == "f32_host":
        return dict(call="f32_host", model=rng.choice(["flat", "volvec"]), paths=_log(rng, 1000, 4194304))
    if call == "philox":
        return dict(call="philox", model=rng.choice(["flat", "volvec"]), paths=_log(rng, 4096, 16777216))
    if call == "curves":
        n = _log(rng, 2, 256)
        return dict(call=rng.choice(["f32", "philox"]), model="curves", curves=n, paths=_log(rng, 256, 4194304 // n))
    if call == "long":
        return dict(call=rng.choice(["f32", "f32", "philox", "pair"]), model="long", paths=_log(rng, 1000, 1048576))
    if call == "shape":
        nn = rng.randrange(16, 257)
        nmat = rng.randrange(4, min(120, nn - 4))
        return dict(call=rng.choice(["f32", "f32", "philox", "pair"]), model="random", nn=nn, nmat=nmat, nopt=rng.randrange(1, 31),
                    paths=_log(rng, 500, 65536))
    if call == "pair":
        return dict(call="pair", model=rng.choice(["flat", "volvec"]), paths=_log(rng, 1000, 1048576))
    if call == "f64":
        if rng.random() < 0.3:
            nn = rng.randrange(16, 201)
            return dict(call="f64", model="random", nn=nn, nmat=rng.randrange(4, min(100, nn - 4)), nopt=rng.randrange(1, 31),
                        paths=_log(rng, 500, 16384))
        return dict(call="f64", model=rng.choice(["flat", "volvec"]), paths=_log(rng, 500, 262144))
    if call == "bump":
        return dict(call="bump", model=rng.choice(["flat", "volvec"]), paths=_log(rng, 256, 16384))
    if call == "entry":
        return dict(call="entry", model="reference", dtype=rng.choice(["f32", "f64"]), paths=_log(rng, 1000, 131072))
    return dict(call="mrg", dtype=rng.choice(["f32", "f64"]), paths=_log(rng, 16384, 4194304))


def _config(case, seed):
    m, paths = case["model"], case["paths"]
    if m == "flat":
        return C.workload(2, paths)
    if m == "reference":
        return C.reference_params(paths)
    if m == "volvec":
        return C.workload(4, paths)
    if m == "long":
        return C.workload(3, paths)
    if m == "curves":
        c = C.workload(5, paths)
        c.L0 = np.ascontiguousarray(c.L0[:case["curves"]])
        return c
    # vols up to 0.2 keep every Euler path tame over these horizons
    rng = np.random.default_rng(seed)
    nn, nmat, nopt = case["nn"], case["nmat"], case["nopt"]
    return C.LmmConfig("random%dx%d" % (nn, nmat), nn, nmat, 0.25, rng.uniform(0.02, 0.07, nn), rng.uniform(0.1, 0.2, nn),
                       rng.integers(1, nn - nmat + 1, nopt).astype(np.int32), rng.uniform(0.03, 0.06, nopt), paths)


def _normals(case, cfg, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float64 if case["call"] in ("f64", "bump") else torch.float32
    return torch.randn(cfg.paths * cfg.nmat, generator=g, device="cuda", dtype=dtype)


def _entry_vol(seed):
    """The entry point takes no seed to any effect: its callers vary mean and standard deviation."""
    return 1.0 + 0.01 * (seed % 17 - 8)


def prepare(case, seed):
    call = case["call"]
    s = dict(case=case, seed=seed)
    if call == "mrg":
        n = case["paths"] * 40
        s["z"] = torch.zeros(n, dtype=torch.float64 if case["dtype"] == "f64" else torch.float32, device="cuda")
        return s
    if call == "entry":
        return s
    cfg = _config(case, seed)
    e = s["engine"] = P.Engine(cfg)
    e.set_stream(torch.cuda.current_stream().cuda_stream)
    if call == "philox":
        pass
    elif call == "f32_host":
        z = torch.empty(cfg.paths * cfg.nmat, dtype=torch.float32, pin_memory=True)
        z.copy_(_normals(case, cfg, seed))
        s["pinned"], s["z"] = z, z.numpy()
    else:
        s["z"] = _normals(case, cfg, seed)
    # value and Greeks, and their standard errors, [2][curves][1 + 2 rates]
    s["out"] = torch.zeros(2, e.nscen, e.nout, dtype=torch.float64, device="cuda")
    if call == "pair":
        s["tape"] = e.tape(cfg.paths)
        s["value"] = torch.zeros(2, e.nscen, dtype=torch.float64, device="cuda")
        s["grad"] = torch.zeros(2, e.nscen, 2 * e.nn, dtype=torch.float64, device="cuda")
    return s


def run(s):
    case, e = s["case"], s.get("engine")
    call, paths = case["call"], case["paths"]
    if call == "mrg":
        fn = P.mrg32k3a_normals_f64_device if case["dtype"] == "f64" else P.mrg32k3a_normals_f32_device
        fn(s["seed"] & 0xFFFFFFFF, 40 * (s["seed"] % 1000003), s["z"].numel(), s["z"].data_ptr(),
           torch.cuda.current_stream().cuda_stream)
        return s["z"]
    if call == "entry":
        fn = P.swaption_greeks if case["dtype"] == "f64" else P.swaption_greeks_f32
        z, v, lb = fn(paths, 0.0, _entry_vol(s["seed"]), rng="mrg32k3a")
        return [z, np.array([v], dtype=z.dtype), np.array([lb], dtype=z.dtype)]
    if call == "f32_host":
        out, se = e.greeks_f32(s["z"], paths)
        return [out.astype(np.float32), se.astype(np.float32)]
    if call == "pair":
        v, g, z = s["value"], s["grad"], s["z"].data_ptr()
        e.forward_f32_device(z, paths, s["tape"], v[0].data_ptr(), v[1].data_ptr())
        e.backward_f32_device(z, s["tape"], [1.0] * e.nscen, g[0].data_ptr(), g[1].data_ptr())
        return [v.float(), g.float()]
    out = s["out"]
    o, se = out.data_ptr(), out.data_ptr() + out[0].numel() * 8
    if call == "f32":
        e.greeks_f32_device(s["z"].data_ptr(), paths, o, se)
        return out.float()
    if call == "philox":
        e.greeks_philox_device(s["seed"], paths, o, se)
        return out.float()
    if call == "f64":
        e.greeks_f64_device(s["z"].data_ptr(), paths, o, se)
        return out
    e.bump_greeks_f64_device(s["z"].data_ptr(), paths, BUMP, o, se)
    return out


def work(case):
    """Reads of the normals and writes of the results; the reference's operations, a divide or an exp counted as one:
    11 per rate and step forward, 12 for the delta sweep, 9 for the vegas, and about 900 for the payoff."""
    call, paths = case["call"], case["paths"]
    if call == "mrg":     # two order-3 recurrences and a rational inversion: about 45 operations for each element
        n = 40 * paths
        return {"bytes": n * (8 if case["dtype"] == "f64" else 4), "flops": 45 * n}
    cfg = _config(case, 0)
    width = 8 if call in ("f64", "bump") or case.get("dtype") == "f64" else 4
    cells = sum(cfg.nn - 1 - n for n in range(cfg.nmat))
    flops = (1 + 2 * cfg.nn) * (11 * cells + 500) if call == "bump" else 32 * cells + 900
    drawn = 45 * cfg.nmat if call in ("entry", "philox") else 0
    nbytes = 16 * cfg.nscen * cfg.nout + (0 if call == "philox" else width * paths * cfg.nmat)
    return {"bytes": nbytes, "flops": cfg.nscen * paths * flops + paths * drawn}


# ---- the same in plain torch, 64 bits ---------------------------------------------------------------------------------


def _payoff(L, cfg, adjoint=True):
    """Discounted portfolio value and (if asked) the log-adjoints L dV/dL of the terminal rates L [paths, nn]."""
    d, nm, M = cfg.delta, cfg.nmat, cfg.nn - cfg.nmat
    r = 1.0 / (1.0 + d * L)
    B = torch.cumprod(r[:, nm:], 1)
    S = d * torch.cumsum(B, 1)
    disc = torch.prod(r[:, :nm], 1)
    val = torch.zeros_like(disc)
    Sb, Bb = torch.zeros_like(B), torch.zeros_like(B)
    for m, k in zip(cfg.maturities.tolist(), cfg.swaprates.tolist()):
        sw = B[:, m - 1] + k * S[:, m - 1] - 1.0
        itm = (sw < 0).to(L.dtype)
        val = val - 100.0 * sw * itm
        if adjoint:
            Sb[:, m - 1] -= 100.0 * k * itm
            Bb[:, m - 1] -= 100.0 * itm
    V = disc * val
    if not adjoint:
        return V, None
    Pb = torch.empty_like(L)
    Pb[:, :nm] = -(V * d)[:, None] * r[:, :nm] * L[:, :nm]
    sb, bb = torch.zeros_like(disc), torch.zeros_like(disc)
    for m in range(M - 1, -1, -1):
        sb = sb + Sb[:, m]
        bb = bb + Bb[:, m] + d * sb
        Pb[:, nm + m] = -disc * bb * B[:, m] * d * r[:, nm + m] * L[:, nm + m]
        bb = bb * r[:, nm + m]
    return V, Pb


def _greeks(cfg, L0, z):
    """[paths, 1 + 2 nn]: value, deltas and vegas of every path, with the reference's recurrences."""
    nn, nm, d = cfg.nn, cfg.nmat, cfg.delta
    lam = torch.as_tensor(cfg.lam, dtype=torch.float64, device=z.device)
    L0 = torch.as_tensor(L0, dtype=torch.float64, device=z.device)
    L = L0.expand(z.shape[0], nn).clone()
    kept = []
    for n in range(nm):
        l, x = lam[: nn - n - 1], math.sqrt(d) * z[:, n: n + 1]
        A = L[:, n + 1:].clone()
        t = A / (1.0 + d * A)
        y = d * torch.cumsum(d * l * t, 1) + x
        kept.append((t, y))
        L[:, n + 1:] = A * torch.exp(l * y - 0.5 * d * l * l)
    V, Pb = _payoff(L, cfg)
    vega = torch.zeros_like(L)
    for n in range(nm - 1, -1, -1):
        l, (t, y) = lam[: nn - n - 1], kept[n]
        pb = Pb[:, n + 1:]
        S = torch.flip(torch.cumsum(torch.flip(l * pb, [1]), 1), [1])
        vega[:, : nn - n - 1] += pb * (y - d * l) + d * d * t * S
        Pb[:, n + 1:] = pb + d * d * l * t * (1.0 - d * t) * S
    return torch.cat([V[:, None], Pb / L0, vega], 1)


def _normals64(case, cfg, seed, first, count):
    """Philox4x32-10 on counters {n/4, 0, path}, 24-bit uniforms, Box-Muller in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nq = (cfg.nmat + 3) // 4
    w = 0xFFFFFFFF
    path = (first + torch.arange(count, dtype=torch.int64, device=dev))[:, None].expand(count, nq)
    c = [torch.arange(nq, dtype=torch.int64, device=dev).expand(count, nq), torch.zeros_like(path), path & w, path >> 32]
    k0, k1 = seed & w, (seed >> 32) & w

    def mul(a, x):
        return ((a * (x >> 16)) + ((a * (x & 0xFFFF)) >> 16)) >> 16, (a * x) & w

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & w, (k1 + 0xBB67AE85) & w
    z = []
    for a, b in ((c[0], c[1]), (c[2], c[3])):
        r = torch.sqrt(-2.0 * torch.log(((a >> 8) + 1).double() / 16777216.0))
        th = 2.0 * math.pi * ((b >> 8).double() / 16777216.0)
        z += [r * torch.cos(th), r * torch.sin(th)]
    return torch.stack(z, 2).reshape(count, 4 * nq)[:, : cfg.nmat]


def _mrg(seed, first, count, mean, sd):
    """Elements first .. first+count-1 of the MRG32k3a stream as normals: sub-streams side by side, all of one length."""
    m1, m2 = 4294967087, 4294944443
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def mul(a, b, m):
        return [[sum(a[i][k] * b[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]

    def power(a, e, m):
        r = [[int(i == j) for j in range(3)] for i in range(3)]
        while e:
            r = mul(r, a, m) if e & 1 else r
            a, e = mul(a, a, m), e >> 1
        return r

    def jump(a, v, m):     # v [3, lanes] int64 below 2^32, entries of a below 2^32: products in 16-bit halves
        return torch.stack([sum((((a[i][k] >> 16) * v[k] % m << 16) + (a[i][k] & 0xFFFF) * v[k]) % m for k in range(3)) % m
                            for i in range(3)])

    A1 = [[0, 1, 0], [0, 0, 1], [m1 - 810728, 1403580, 0]]
    A2 = [[0, 1, 0], [0, 0, 1], [m2 - 1370589, 0, 527612]]
    lanes = 1 << 17
    span = max(1, -(-count // lanes))
    X = torch.tensor([[seed % m1], [1], [1]], dtype=torch.int64, device=dev)
    Y = torch.ones(3, 1, dtype=torch.int64, device=dev)
    X, Y = jump(power(A1, first, m1), X, m1), jump(power(A2, first, m2), Y, m2)
    while X.shape[1] < lanes:
        s = span * X.shape[1]
        X = torch.cat([X, jump(power(A1, s, m1), X, m1)], 1)
        Y = torch.cat([Y, jump(power(A2, s, m2), Y, m2)], 1)
    x, y = list(X), list(Y)
    out = torch.empty(span, lanes, dtype=torch.float64, device=dev)
    for k in range(span):
        p, q = (1403580 * x[1] - 810728 * x[0]) % m1, (527612 * y[2] - 1370589 * y[0]) % m2
        x, y = [x[1], x[2], p], [y[1], y[2], q]
        u = torch.where(p > q, p - q, p - q + m1)
        # the upper half through the lower tail, where 1 - u would round
        low = torch.minimum(u, m1 + 1 - u).double() / (m1 + 1)
        out[k] = mean + sd * torch.special.ndtri(low) * torch.where(u * 2 > m1 + 1, -1.0, 1.0)
    return out.t().reshape(-1)[:count]


def _mean_se(total, square, n):
    mu = total / n
    var = ((square - total * mu) / (n - 1)).clamp(min=0.0) if n > 1 else torch.zeros_like(mu)
    return mu, torch.sqrt(var / n)


def exact(case, seed):
    call, paths = case["call"], case["paths"]
    if call == "mrg":
        return _mrg(seed & 0xFFFFFFFF, 40 * (seed % 1000003), 40 * paths, 0.0, 1.0)
    cfg = _config(case, seed)
    nn, nm, nout = cfg.nn, cfg.nmat, cfg.nout
    curves = np.atleast_2d(cfg.L0)
    z = None
    if call == "entry":
        z = _mrg(12345, 0, nm * paths, 0.0, _entry_vol(seed)).reshape(paths, nm)
    elif call != "philox":
        z = _normals(case, cfg, seed).reshape(paths, nm)
    if call == "bump":
        z = z.double()
        var = [(curves[0], cfg.lam)]
        var += [(curves[0] + BUMP * np.eye(nn)[j], cfg.lam) for j in range(nn)]
        var += [(curves[0], cfg.lam + BUMP * np.eye(nn)[j]) for j in range(nn)]
        res = torch.zeros(2, 1, nout, dtype=torch.float64)
        for j, (L0, lam) in enumerate(var):
            l = torch.as_tensor(lam, dtype=torch.float64, device=z.device)
            L = torch.as_tensor(L0, dtype=torch.float64, device=z.device).expand(paths, nn).clone()
            for n in range(nm):
                A, ln = L[:, n + 1:], l[: nn - n - 1]
                v = torch.cumsum(cfg.delta * ln * A / (1.0 + cfg.delta * A), 1)
                L[:, n + 1:] = A * torch.exp(ln * (cfg.delta * v + math.sqrt(cfg.delta) * z[:, n: n + 1] - 0.5 * cfg.delta * ln))
            V, _ = _payoff(L, cfg, adjoint=False)
            mu, se = _mean_se(V.sum(), V.square().sum(), paths)
            if j == 0:
                base, res[0, 0, 0], res[1, 0, 0] = mu, mu, se
            else:
                res[0, 0, j] = (mu - base) / BUMP
        return res
    chunk = max(1, int(2e9 // (16 * nn * nm)))
    mean, err = [], []
    for L0 in curves:
        total, square = 0.0, 0.0
        for first in range(0, paths, chunk):
            n = min(chunk, paths - first)
            zc = _normals64(case, cfg, seed, first, n) if z is None else z[first: first + n].double()
            g = _greeks(cfg, L0, zc)
            total, square = total + g.sum(0), square + g.square().sum(0)
        mu, se = _mean_se(total, square, paths)
        mean.append(mu)
        err.append(se)
    mean, err = torch.stack(mean), torch.stack(err)
    if call == "entry":
        return [z.reshape(-1), mean[0, :1], mean[0, nn: nn + 1]]
    if call == "f32_host":
        return [mean, err]
    if call == "pair":
        return [torch.stack([mean[:, 0], err[:, 0]]), torch.stack([mean[:, 1:], err[:, 1:]])]
    return torch.stack([mean, err])
