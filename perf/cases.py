"""Performance cases of the transform paths: sizes, inputs and one pass of each.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` builds what a program holds before the call (inputs on the GPU or
in host arrays, output buffers, parameters, the context), ``run`` is one pass
through the public entry points, ``work`` counts what a pass cannot do without
and ``exact`` computes the same outputs in 64-bit torch without this library.

A case is a dict of plain values:

  kind        "single"   so3gpu context calls on one signal (device buffers)
              "batch"    inverse_batch / forward_batch, `count` signals
              "ragged"   inverse_ragged / forward_ragged, `count` signals whose
                         sizes come from `shapes` (a seed), L up to `L`
              "conv"     s2toso3_inverse_batch: one S^2 signal, `count` kernels
              "host"     the numpy drop-in calls so3.inverse / so3.forward
              "adjoint"  the numpy calls so3.adjoint_inverse / adjoint_forward
  dir         "inverse", "forward" or "both"
  L, N, L0    band limits
  real, mwss, compact, zero_first, n_mode, trapani, steerable   parameter flags
  precision   "fp64" or "mixed" (batch, ragged, conv)
  dist        coefficients "uniform" (U(-1,1)) or "gauss" (variance (l+1)^-2)
"""
import math
import random

import torch

import so3_b200 as so3

_DEFAULTS = dict(kind="single", dir="both", L=16, N=4, L0=0, real=False, mwss=False, compact=False, zero_first=False,
                 n_mode=0, trapani=False, steerable=False, count=1, precision="fp64", dist="uniform", shapes=0)
_SERVED_L = 512          # split-precision reach of the request server
_MOST = 512 ** 3 * 64    # L^3 N of the largest single transform


def listed():
    return [
        # The smallest call: a low-resolution signal in an interactive or optimisation loop (launch latency).
        dict(name="small L16 N4", kind="single", L=16, N=4),
        # The plain complex round trip at L = N = 64 of the configurations.
        dict(name="complex L64 N64", kind="single", L=64, N=64),
        # Real signals on the equiangular MWSS grid, compact storage, Trapani recursion.
        dict(name="real MWSS L256 N32", kind="single", L=256, N=32, real=True, mwss=True, compact=True, trapani=True,
             dist="gauss"),
        # The headline geometry, one signal per call in FP64.
        dict(name="fp64 L512 N64", kind="single", L=512, N=64),
        # An odd band limit (2L-1 = 599 is prime), even n only, compact and zero-first.
        dict(name="odd L300 N21 even n", kind="single", L=300, N=21, compact=True, zero_first=True, n_mode=1,
             dist="gauss"),
        # The headline batch in split precision, one case per direction.
        dict(name="split inverse L512 N64 x16", kind="batch", dir="inverse", L=512, N=64, count=16,
             precision="mixed"),
        dict(name="split forward L512 N64 x16", kind="batch", dir="forward", L=512, N=64, count=16,
             precision="mixed"),
        # Many mid-size signals in split precision (Monte-Carlo sets, training batches).
        dict(name="split L128 N16 x128", kind="batch", L=128, N=16, count=128, precision="mixed", dist="gauss"),
        # Directional convolution of one high-resolution sky with eight directional kernels, FP64.
        dict(name="conv L1024 N8 x8", kind="conv", L=1024, N=8, count=8, dist="gauss"),
        # A unit of the serving trace: requests of mixed sizes that share tensor-core tiles.
        dict(name="ragged split x16", kind="ragged", L=_SERVED_L, N=64, count=16, precision="mixed", shapes=3),
        # The drop-in calls on numpy arrays, as a relinked CPU program makes them.
        dict(name="host L128 N8", kind="host", L=128, N=8),
        # Adjoints of both transforms on numpy arrays (gradients of inverse problems).
        dict(name="adjoint L96 N12", kind="adjoint", L=96, N=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single"] * 6 + ["batch"] * 3 + ["ragged", "conv", "host", "adjoint"])
    c = dict(kind=kind, dist=rng.choice(["uniform", "gauss"]))
    if kind == "single":
        c["L"] = _log_int(rng, 16, 1024)
        c["N"] = rng.randint(1, max(1, min(c["L"], 64, _MOST // c["L"] ** 3)))
        c["dir"] = rng.choice(["inverse", "forward", "both"])
        c.update(mwss=rng.random() < 0.25, compact=rng.random() < 0.3, zero_first=rng.random() < 0.2,
                 n_mode=rng.choice([0, 0, 0, 0, 1, 2, 3]), trapani=rng.random() < 0.3, L0=rng.choice([0, 0, 0, 1, 2]))
        if rng.random() < 0.3 and c["N"] > 1:
            c["real"], c["zero_first"] = True, False
        elif rng.random() < 0.15:
            c["steerable"] = True
        if c["N"] == 1 or c.get("steerable"):
            c["n_mode"] = 0  # the other modes could leave no coefficient
    elif kind == "batch":
        c["L"] = _log_int(rng, 16, _SERVED_L)
        c["N"] = rng.randint(2, min(c["L"], 64))
        room = _MOST // (c["L"] ** 3 * c["N"])
        c["count"] = rng.randint(1, max(1, min(64, room * 8)))
        c["precision"] = rng.choice(["mixed", "mixed", "fp64"])
        c["dir"] = rng.choice(["inverse", "forward", "both"])
        c["real"] = rng.random() < 0.2
    elif kind == "ragged":
        c.update(L=_log_int(rng, 64, _SERVED_L), N=rng.randint(4, 32), count=rng.randint(2, 24),
                 shapes=rng.randrange(1 << 20), precision="mixed", dir=rng.choice(["inverse", "forward", "both"]))
    elif kind == "conv":
        c["L"] = _log_int(rng, 32, 1024)
        c["N"] = rng.randint(1, min(c["L"], 16))
        c["count"] = max(1, min(rng.randint(1, 16), (8 * 8 * 1024 ** 3) // (c["L"] ** 3 * c["N"])))
        c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
    elif kind == "host":
        c["L"] = _log_int(rng, 16, 256)
        c["N"] = rng.randint(1, min(c["L"], 16))
        c["dir"] = rng.choice(["inverse", "forward", "both"])
    else:
        c["L"] = _log_int(rng, 16, 256)
        c["N"] = rng.randint(1, min(c["L"], 16))
        c["real"] = rng.random() < 0.3 and c["N"] > 1
    return c


# ------------------------------------------------------------------ parameters and layouts
def _params(c):
    return so3.SO3Parameters(L=c["L"], N=c["N"], L0=c["L0"], reality=int(c["real"]), sampling_scheme=int(c["mwss"]),
                             n_order=0 if c["zero_first"] else 1, storage=int(c["compact"]), n_mode=c["n_mode"],
                             dl_method=int(c["trapani"]), steerable=int(c["steerable"]))


def _full(case):
    return {**_DEFAULTS, **case}


def _signals(c):
    """One case dict per signal of a pass (ragged batches: its own sizes each)."""
    if c["kind"] != "ragged":
        return [c] * c["count"]
    rng = random.Random(c["shapes"])
    out = []
    for _ in range(c["count"]):
        L = _log_int(rng, 16, c["L"])
        out.append({**c, "L": L, "N": rng.randint(1, min(L, c["N"]))})
    return out


def _planes(c):
    """n of the coefficient blocks in storage order."""
    N = c["N"]
    if c["real"]:
        return list(range(N))
    if c["zero_first"]:
        return [0] + [s * n for n in range(1, N) for s in (-1, 1)]
    return list(range(-(N - 1), N))


def _active(c, n):
    if c["n_mode"] == 1:
        return n % 2 == 0
    if c["n_mode"] == 2:
        return n % 2 != 0
    if c["n_mode"] == 3:
        return abs(n) >= c["N"] - 1
    return True


def _grid(c):
    """(gamma, beta, alpha) samples."""
    L = c["L"]
    return (c["N"] if c["steerable"] else 2 * c["N"] - 1), (L + 1 if c["mwss"] else L), (2 * L if c["mwss"] else 2 * L - 1)


def _flmn_size(c):
    return sum(c["L"] ** 2 - (n * n if c["compact"] else 0) for n in _planes(c))


def _f_size(c):
    g = _grid(c)
    return g[0] * g[1] * g[2]


def _el_m(L, dev):
    e = torch.arange(L * L, device=dev)
    el = torch.sqrt(e.double()).floor().long()
    el = torch.where(el * el > e, el - 1, el)
    el = torch.where((el + 1) * (el + 1) <= e, el + 1, el)
    return el, e - el * el - el


def _noise(count, c, el, gen, dev):
    if c["dist"] == "uniform":
        return torch.view_as_complex(torch.rand(count, 2, dtype=torch.float64, device=dev, generator=gen) * 2 - 1)
    v = torch.view_as_complex(torch.randn(count, 2, dtype=torch.float64, device=dev, generator=gen))
    return v / (math.sqrt(2.0) * (el + 1))


def _coefficients(c, gen, dev, out):
    """Random coefficients of one signal in its own layout, l >= max(L0, |n|)
    of the n the n-mode keeps, zero elsewhere."""
    L = c["L"]
    el, m = _el_m(L, dev)
    at = 0
    for n in _planes(c):
        cut = n * n if c["compact"] else 0
        v = _noise(L * L, c, el, gen, dev)
        if c["real"] and n == 0:  # f_{l,-m,0} = (-1)^m conj f_{l,m,0}
            w = v[el * el + el + m.abs()]
            v = torch.where(m < 0, torch.where(m % 2 != 0, -1.0, 1.0).double() * w.conj(), w)
            v = torch.where(m == 0, v.real.to(v.dtype), v)
        v = v * ((el >= max(c["L0"], abs(n))) & _active(c, n))
        out[at:at + L * L - cut] = v[cut:]
        at += L * L - cut


def _samples(c, gen, dev, out):
    """Random samples of one signal (noise maps: not band-limited)."""
    (out if c["real"] else torch.view_as_real(out)).normal_(generator=gen)


def _inputs(c, seed, dev):
    """{"flmn": [...], "f": [...]} or {"flm", "glm"}: views of one tensor per kind."""
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 1000003 + 17)
    if c["kind"] == "conv":
        el, m = _el_m(c["L"], dev)
        sky = lambda: _noise(c["L"] ** 2, {"dist": "gauss"}, el, gen, dev)  # noqa: E731
        return {"flm": sky(), "glm": [sky() * (m.abs() < c["N"]) for _ in range(c["count"])]}
    sig, got = _signals(c), {}
    for what, size, fill in (("flmn", _flmn_size, _coefficients), ("f", _f_size, _samples)):
        if c["kind"] != "adjoint" and c["dir"] == ("forward" if what == "flmn" else "inverse"):
            continue
        dt = torch.float64 if what == "f" and c["real"] else torch.complex128
        whole = torch.empty(sum(size(s) for s in sig), dtype=dt, device=dev)
        got[what] = list(whole.split([size(s) for s in sig]))
        for s, x in zip(sig, got[what]):
            fill(s, gen, dev, x)
    return got


# ------------------------------------------------------------------ the calls
_context = None


def _ctx():
    """The one context that a program keeps for its stream."""
    global _context
    if _context is None:
        _context = so3.Context(0)
    return _context


def _outputs(sizes, dtype):
    """Zeroed output buffers: the first signal's and the others' (one tensor
    each), and the list of all of them."""
    first = torch.zeros(sizes[0], dtype=dtype, device="cuda")
    rest = torch.zeros(sum(sizes[1:]), dtype=dtype, device="cuda")
    return first, rest, [first] + (list(rest.split(sizes[1:])) if len(sizes) > 1 else [])


def prepare(case, seed):
    c = _full(case)
    x = _inputs(c, seed, "cuda")
    st = {"c": c, "p": _params(c)}
    if c["kind"] in ("host", "adjoint"):
        for k, v in x.items():
            st[k] = v[0].cpu().numpy()
        return st
    sig = _signals(c)
    st.update(x, ctx=_ctx(), ps=[_params(s) for s in sig])
    for p in {(s["L"], s["N"]): p for s, p in zip(sig, st["ps"])}.values():
        st["ctx"].prepare(p)
    if "flmn" in x or "flm" in x:
        st["f_out"] = _outputs([_f_size(s) for s in sig], torch.float64 if c["real"] else torch.complex128)
    if "f" in x:
        st["flmn_out"] = _outputs([_flmn_size(s) for s in sig], torch.complex128)
    return st


def run(st):
    c, p, out = st["c"], st["p"], {}
    kind = c["kind"]
    if kind == "host":
        if "flmn" in st:
            out["f"] = so3.inverse(st["flmn"], p)
        if "f" in st:
            out["flmn"] = so3.forward(st["f"], p)
        return out
    if kind == "adjoint":
        return {"flmn": so3.adjoint_inverse(st["f"], p), "f": so3.adjoint_forward(st["flmn"], p)}
    ctx = st["ctx"]
    if kind == "conv":
        ctx.s2toso3_inverse_batch(p, st["flm"], st["glm"], c["precision"], outs=st["f_out"][2])
    elif kind == "single":
        if "f_out" in st:
            ctx.inverse(st["flmn"][0], p, out=st["f_out"][0])
        if "flmn_out" in st:
            ctx.forward(st["f"][0], p, out=st["flmn_out"][0])
    elif kind == "batch":
        if "f_out" in st:
            ctx.inverse_batch(st["flmn"], p, c["precision"], outs=st["f_out"][2])
        if "flmn_out" in st:
            ctx.forward_batch(st["f"], p, c["precision"], outs=st["flmn_out"][2])
    else:
        if "f_out" in st:
            ctx.inverse_ragged(st["flmn"], st["ps"], c["precision"], outs=st["f_out"][2])
        if "flmn_out" in st:
            ctx.forward_ragged(st["f"], st["ps"], c["precision"], outs=st["flmn_out"][2])
    if "f_out" in st:
        out["f"] = list(st["f_out"][:2])
    if "flmn_out" in st:
        out["flmn"] = list(st["flmn_out"][:2])
    return out


# ------------------------------------------------------------------ work
def _one_way(s):
    """(coefficient bytes, sample bytes, flops) of one transform of signal s:
    the Delta products (a complex times a real) over every coefficient and
    0 <= m' <= l, and the DFTs over the three angles."""
    planes = [n for n in _planes(s) if _active(s, n)]
    g, b, a = _grid(s)

    def products(k):  # sum over l < k of (2l+1)(l+1)
        return k * (k - 1) * (2 * k - 1) / 3 + 3 * k * (k - 1) / 2 + k

    def dft(n):
        return 5.0 * n * math.log2(max(n, 2))

    flops = sum(4.0 * max(0.0, products(s["L"]) - products(max(abs(n), s["L0"]))) for n in planes)
    flops += len(planes) * (a * dft(a) / 2 + b * dft(a)) + a * b * dft(2 * s["N"] - 1) / (2 if s["real"] else 1)
    return 16.0 * _flmn_size(s), (8.0 if s["real"] else 16.0) * _f_size(s), flops


def work(case):
    c = _full(case)
    ways = 2 if c["kind"] == "adjoint" or c["dir"] == "both" else 1
    total = {"bytes": 0.0, "flops": 0.0}
    if c["kind"] == "conv":
        total["bytes"] += 16.0 * c["L"] ** 2
        ways = 1
    for s in _signals(c):
        cb, fb, fl = _one_way(s)
        total["bytes"] += fb + 16.0 * s["L"] ** 2 if c["kind"] == "conv" else ways * (cb + fb)
        total["flops"] += ways * fl
    return total


# ------------------------------------------------------------------ exact values
def _deltas(L, dev):
    """Delta^l = d^l(pi/2), rows and columns -l..l, for l = 0..L-1 in turn, by
    the half-degree recursion of Risbo (1996) at cos = sin = 1/sqrt 2."""
    d = torch.ones(1, 1, dtype=torch.float64, device=dev)
    yield d
    for l in range(1, L):
        for j in (2 * l - 1, 2 * l):
            down = torch.sqrt(torch.arange(j, 0, -1, dtype=torch.float64, device=dev))
            up = torch.sqrt(torch.arange(1, j + 1, dtype=torch.float64, device=dev))
            s = d * (math.sqrt(0.5) / j)
            d = torch.zeros(j + 1, j + 1, dtype=torch.float64, device=dev)
            d[:j, :j] += down[:, None] * down[None, :] * s
            d[1:, :j] -= up[:, None] * down[None, :] * s
            d[:j, 1:] += down[:, None] * up[None, :] * s
            d[1:, 1:] += up[:, None] * up[None, :] * s
        yield d


def _i_pow(k, dev):
    return torch.tensor([1, 1j, -1, -1j], dtype=torch.complex128, device=dev)[k % 4]


def _unpack(c, x):
    """Coefficient layout -> [plane in _planes order, L^2], l < |n| zero."""
    L, rows, at = c["L"], [], 0
    for n in _planes(c):
        cut = n * n if c["compact"] else 0
        r = torch.zeros(L * L, dtype=torch.complex128, device=x.device)
        r[cut:] = x[at:at + L * L - cut]
        rows.append(r)
        at += L * L - cut
    return torch.stack(rows)


def _pack(c, rows):
    return torch.cat([r[n * n if c["compact"] else 0:] for n, r in zip(_planes(c), rows)])


def _spectra(c, coef, weight):
    """[plane, L^2] -> F[plane, m' >= 0, m + L - 1] = i^{n-m} sum_l weight(l)
    Delta^l_{m'm} Delta^l_{m'n} coef."""
    L, dev, planes = c["L"], coef.device, _planes(c)
    F = torch.zeros(len(planes), L, 2 * L - 1, dtype=torch.complex128, device=dev)
    ns = torch.tensor(planes, device=dev)
    for l, d in enumerate(_deltas(L, dev)):
        keep = (ns.abs() <= l).nonzero().flatten()
        v = coef[keep, l * l:(l + 1) ** 2] * weight(l)
        both = d[l:, :][:, ns[keep] + l].T[:, :, None] * d[l:, :][None]  # [plane, m', m]
        F[keep, :l + 1, L - 1 - l:L + l] += v[:, None, :] * both
    m = torch.arange(-(L - 1), L, device=dev)
    return F * _i_pow(ns[:, None] - m[None, :], dev)[:, None, :]


def _contract(c, G, weight):
    """G[plane, m' >= 0 (folded), m + L - 1] -> [plane, L^2]: i^{m-n} sum_{m'=0}^l
    weight(l) Delta Delta G; entries l < max(L0, |n|) and skipped planes zero."""
    L, dev, planes = c["L"], G.device, _planes(c)
    ns = torch.tensor(planes, device=dev)
    out = torch.zeros(len(planes), L * L, dtype=torch.complex128, device=dev)
    live = torch.tensor([_active(c, n) for n in planes], device=dev)
    for l, d in enumerate(_deltas(L, dev)):
        if l < c["L0"]:
            continue
        keep = ((ns.abs() <= l) & live).nonzero().flatten()
        m = torch.arange(-l, l + 1, device=dev)
        both = d[l:, :][:, ns[keep] + l].T[:, :, None] * d[l:, :][None]
        v = (G[keep, :l + 1, L - 1 - l:L + l] * both).sum(1)
        out[keep, l * l:(l + 1) ** 2] = v * _i_pow(m[None, :] - ns[keep][:, None], dev) * weight(l)
    return out


def _signs(c, dev):
    """(-1)^{m+n} over [plane, 1, m + L - 1]."""
    ns = torch.tensor(_planes(c), device=dev)
    m = torch.arange(-(c["L"] - 1), c["L"], device=dev)
    return torch.where((ns[:, None] + m[None, :]) % 2 == 0, 1.0, -1.0).double()[:, None, :]


def _orders(c, dev):
    return torch.arange(-(c["L"] - 1), c["L"], device=dev, dtype=torch.float64)


def _betas(c, dev):
    k = torch.arange(_grid(c)[1], device=dev, dtype=torch.float64)
    return math.pi * k / c["L"] if c["mwss"] else math.pi * (2 * k + 1) / (2 * c["L"] - 1)


def _analysis(c, s, dev):
    """K_s [m' = -(L-1)..L-1, beta]: beta samples extended onto the circle with
    parity s, their spectrum over m'', and the integral over theta of
    e^{i(m'' - m') theta} sin(theta)."""
    L, mw = c["L"], not c["mwss"]
    P, nb = _grid(c)[2], _grid(c)[1]
    t = torch.arange(P, device=dev, dtype=torch.float64)
    th = math.pi * (2 * t + 1) / P if mw else 2 * math.pi * t / P
    E = torch.exp(-1j * _orders(c, dev)[:, None] * th[None, :]) / P
    V = E[:, :nb].clone()
    for r in range(nb, P):  # row r of the circle mirrors a sampled row
        V[:, 2 * L - 2 - r if mw else 2 * L - r] += s * E[:, r]
    p = torch.arange(-2 * (L - 1), 2 * (L - 1) + 1, device=dev)
    w = torch.where(p % 2 == 0, 2.0 / (1.0 - p.double() ** 2), torch.zeros_like(p).double()).to(torch.complex128)
    w += 1j * math.pi / 2 * ((p == 1).double() - (p == -1).double())
    d = torch.arange(2 * L - 1, device=dev)
    return 2 * math.pi * w[d[None, :] - d[:, None] + 2 * (L - 1)] @ V


def _fold(c, X):
    """[plane, m' = -(L-1)..L-1, m] -> G(m') + (-1)^{m+n} G(-m'), m' >= 0."""
    L = c["L"]
    G = X[:, L - 1:, :].clone()
    G[:, 1:, :] += _signs(c, X.device) * X[:, :L - 1, :].flip(1)
    return G


def _two_sided(c, F):
    """m' >= 0 -> m' = -(L-1)..L-1 with F(-m') = (-1)^{m+n} F(m')."""
    return torch.cat([(_signs(c, F.device) * F[:, 1:, :]).flip(1), F], 1)


def _by_parity(c, X, build):
    """Applies the matrix build(s) over the middle axis to the columns of parity s."""
    sg = _signs(c, X.device)
    return sum(torch.matmul(build(s), X * (sg == s)) for s in (1, -1))


def _angles(c, X):
    """[plane, beta, m] -> samples f[gamma, beta, alpha]: sums over m and n."""
    g, b, a = _grid(c)
    Y = torch.zeros(X.shape[0], b, a, dtype=X.dtype, device=X.device)
    Y[:, :, _orders(c, X.device).long() % a] = X
    Y = torch.fft.ifft(Y, dim=2) * a
    ng = 2 * c["N"] if c["steerable"] else g
    Z = torch.zeros(ng, b, a, dtype=X.dtype, device=X.device)
    for i, n in enumerate(_planes(c)):
        Z[n % ng] = Y[i]
        if c["real"]:  # planes n >= 0 of a real signal
            Z[-n % ng] = Y[i].conj() if n else Y[i].real.to(Y.dtype)
    f = (torch.fft.ifft(Z, dim=0) * ng)[:g].reshape(-1)
    return f.real.contiguous() if c["real"] else f


def _spectral(c, f):
    """samples -> [plane, beta, m], sums of f e^{-i m alpha - i n gamma}."""
    g, b, a = _grid(c)
    ng = 2 * c["N"] if c["steerable"] else g
    Z = torch.zeros(ng, b, a, dtype=torch.complex128, device=f.device)
    Z[:g] = f.reshape(g, b, a)
    Z = torch.fft.fft(Z, dim=0)
    Z = torch.stack([Z[n % ng] for n in _planes(c)])
    return torch.fft.fft(Z, dim=2)[:, :, _orders(c, f.device).long() % a]


def _inverse(c, flmn):
    F = _two_sided(c, _spectra(c, _unpack(c, flmn), lambda l: (2 * l + 1) / (8 * math.pi ** 2)))
    return _angles(c, torch.exp(1j * _betas(c, F.device)[:, None] * _orders(c, F.device)[None, :]) @ F)


def _forward(c, f):
    g, _, a = _grid(c)
    X = _spectral(c, f) * (2 * math.pi / g / a)
    if c["steerable"]:  # only n = N-1 (mod 2) is analysed
        for i, n in enumerate(_planes(c)):
            if (n - (c["N"] - 1)) % 2:
                X[i] = 0
    G = _by_parity(c, X, lambda s: _analysis(c, s, f.device))
    return _pack(c, _contract(c, _fold(c, G), lambda l: 1.0))


def _adjoint_inverse(c, f):
    X = _spectral(c, f)
    G = torch.exp(-1j * _orders(c, f.device)[:, None] * _betas(c, f.device)[None, :]) @ X
    return _pack(c, _contract(c, _fold(c, G), lambda l: (2 * l + 1) / (8 * math.pi ** 2)))


def _adjoint_forward(c, flmn):
    g, _, a = _grid(c)
    F = _two_sided(c, _spectra(c, _unpack(c, flmn), lambda l: 1.0))
    X = _by_parity(c, F, lambda s: _analysis(c, s, F.device).conj().T)
    return _angles(c, X * (2 * math.pi / g / a))


def exact(case, seed):
    c = _full(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = _inputs(c, seed, dev)
    s = _signals(c)[0]
    if c["kind"] == "conv":
        l = torch.arange(c["L"], device=dev)
        rows = []
        for n in _planes(c):
            g = torch.zeros(c["L"], dtype=torch.complex128, device=dev)
            k = l[abs(n):]
            g[abs(n):] = x["glm"][0][k * k + k + n].conj() * (8 * math.pi ** 2) / (2 * k + 1)
            rows.append(x["flm"] * g[_el_m(c["L"], dev)[0]])
        return {"f": [_inverse(s, _pack(s, rows)), None]}
    if c["kind"] == "adjoint":
        out = {"flmn": _adjoint_inverse(s, x["f"][0]), "f": _adjoint_forward(s, x["flmn"][0])}
        return {k: v.cpu().numpy() for k, v in out.items()}
    out = {}
    if "flmn" in x:
        out["f"] = _inverse(s, x["flmn"][0])
    if "f" in x:
        out["flmn"] = _forward(s, x["f"][0])
    if c["kind"] == "host":
        return {k: v.cpu().numpy() for k, v in out.items()}
    return {k: [v, None] for k, v in out.items()}
