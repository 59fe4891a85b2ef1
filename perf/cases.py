"""The work this library does for its users, as cases that can be timed and compared.

Every case names a lattice (nx, ny, nz, nt), what is applied to it (`kind`) and the options of that call.  Inputs are
made from the seed with torch alone: thin SU(3) links close to the identity with the staggered phases folded in, fat
links 9/8 U plus a non-unitary part (fat links are sums of smeared paths), Naik links -1/24 U(x) U(x+mu) U(x+2mu),
Gaussian sources, mass 0.05 and shifts log-spaced 1e-4..1.  `exact` restates the operator, the multishift CG and the
preconditioner network in 64-bit torch on gathered neighbours.

Fields live on the checkerboard: i = (x >> 1) + nx/2 (y + ny (z + nz t)), x = 2 (i mod nx/2) + ((y + z + t + p) & 1).
"""
import math

import numpy as np
import torch

import kuqcd_b200 as K

MASS2 = 0.05 ** 2
SMIN = 1e-4
RES = 1e-10
EPS = 0.25       # width of the thin links around the identity
FAT_NOISE = 0.02  # non-unitary part of the fat links
CHANNELS = (1, 8, 8)
PREC = {64: K.KUQCD_DOUBLE, 32: K.KUQCD_SINGLE, 16: K.KUQCD_HALF}
# CG iterations to 1e-10 at this mass and these shifts, as counted on 16^4 .. 32^4 (they hardly depend on the size)
ITERS = 300


def case(kind, dims, **more):
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "nt": dims[3]}
    c.update(more)
    return c


def listed():
    return [
        # one operator application in a caller's own Krylov loop on the smallest lattice: launches and latency
        case("op", (8, 8, 8, 8), prec=64, name="op64_8x8x8x8"),
        # the same on the largest lattice this library is benchmarked on: memory bandwidth
        case("op", (48, 48, 48, 96), prec=64, name="op64_48x48x48x96"),
        # the 16-bit operator inside a caller's mixed-precision loop (the decomposed-lattice solver's form): vector
        # to 16 bits, operator, result back to 32 bits
        case("op", (32, 32, 32, 32), prec=16, name="op16_32x32x32x32"),
        # the operator without even-odd preconditioning, 32 bits, on a ragged lattice with an odd extent
        case("full", (20, 18, 15, 30), prec=32, name="full32_20x18x15x30"),
        # the drop-in call on the smallest lattice: host arrays in and out, the reference's FP64 multishift CG
        case("solve", (8, 8, 8, 8), solver="cgm", host=True, shifts=12, name="solve_cgm_host_8x8x8x8"),
        # mixed-precision multishift solve, a lattice whose links fit in the L2
        case("solve", (16, 16, 16, 16), solver="mixed", host=False, shifts=12, name="solve_mixed_16x16x16x16"),
        # the reference-order FP64 multishift CG on an ordinary lattice with device fields
        case("solve", (24, 24, 24, 48), solver="cgm", host=False, shifts=12, name="solve_cgm_24x24x24x48"),
        # the mixed-precision multishift solve the library is tuned for
        case("solve", (32, 32, 32, 32), solver="mixed", host=False, shifts=12, name="solve_mixed_32x32x32x32"),
        # the check after a solve: FP64 true residuals of every shift's solution
        case("residuals", (24, 24, 24, 48), shifts=12, name="residuals_24x24x24x48"),
        # propagator sources on one gauge field, solved together
        case("batch", (16, 16, 16, 16), sources=8, shifts=8, name="batch_8x16x16x16x16"),
        # the learned preconditioner: one application, and one training pair (forward, loss and weight gradient)
        case("net", (32, 32, 32, 32), train=False, name="net_apply_32x32x32x32"),
        case("net", (16, 16, 16, 16), train=True, name="net_train_16x16x16x16"),
    ]


def draw(rng):
    kind = rng.choice(["op", "op", "full", "solve", "solve", "residuals", "batch", "net"])
    top = {"op": 32, "full": 28, "solve": 24, "residuals": 24, "batch": 16, "net": 24}[kind]
    size = lambda: int(round(math.exp(rng.uniform(math.log(6), math.log(top)))))  # noqa: E731
    dims = (2 * max(2, size() // 2), size(), size(), size())
    if kind in ("op", "full"):
        return case(kind, dims, prec=rng.choice([64, 32, 16] if kind == "op" else [64, 32]))
    # the solvers run on even-odd lattices in earnest: even extents
    dims = tuple(2 * (n // 2) for n in dims)
    if kind == "solve":
        return case(kind, dims, solver=rng.choice(["cgm", "mixed"]), host=rng.random() < 0.3,
                    shifts=rng.choice([1, 4, 9, 12, 16]))
    if kind == "residuals":
        return case(kind, dims, shifts=rng.choice([1, 3, 8, 12, 16]))
    if kind == "batch":
        return case(kind, dims, sources=rng.choice([3, 4, 8]), shifts=rng.choice([4, 8]))
    return case(kind, dims, train=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------------- inputs
def dims_of(c):
    return c["nx"], c["ny"], c["nz"], c["nt"]


def volume(c):
    return c["nx"] * c["ny"] * c["nz"] * c["nt"]


def sigmas(c):
    n = c.get("shifts", 1)
    return [MASS2 + s for s in (np.logspace(math.log10(SMIN), 0, n) if n > 1 else [SMIN])]


def generator(seed, which):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) % (1 << 40)) + which)
    return g


def gauss(shape, g):
    return torch.view_as_complex(torch.randn(*shape, 2, dtype=torch.float64, device="cuda", generator=g))


def by_parity(f):
    """[nt, nz, ny, nx, ...] lexicographic -> [2, Vh, ...] checkerboard."""
    nt, nz, ny, nx = f.shape[:4]
    h = f.reshape(nt, nz, ny, nx // 2, 2, *f.shape[4:])
    t, z, y = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (nt, nz, ny)), indexing="ij")
    even = ((t + z + y) % 2 == 0).reshape(nt, nz, ny, 1, *([1] * (f.dim() - 4)))
    a, b = h[:, :, :, :, 0], h[:, :, :, :, 1]
    return torch.stack([torch.where(even, a, b).flatten(0, 3), torch.where(even, b, a).flatten(0, 3)])


def links(c, seed):
    """Per direction (fat, long) as [2, Vh, 3, 3] complex128, without the operator's own factors."""
    nx, ny, nz, nt = dims_of(c)
    coord = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (nt, nz, ny, nx)), indexing="ij")[::-1]
    for mu in range(4):
        g = generator(seed, mu)
        a = EPS * gauss((nt, nz, ny, nx, 3), g)
        b = EPS * gauss((nt, nz, ny, nx, 3), g)
        a[..., 0] += 1
        b[..., 1] += 1
        a /= a.abs().square().sum(-1, keepdim=True).sqrt()
        b -= (a.conj() * b).sum(-1, keepdim=True) * a
        b /= b.abs().square().sum(-1, keepdim=True).sqrt()
        u = torch.stack([a, b, torch.linalg.cross(a, b).conj()], -2)
        eta = 1.0 - 2.0 * (sum(coord[:mu], torch.zeros_like(coord[0])) % 2).double()[..., None, None]
        axis = 3 - mu
        prod = u
        for hop in (1, 2):
            nxt = torch.roll(u, -hop, axis)
            prod = sum(prod[..., :, k, None] * nxt[..., None, k, :] for k in range(3))
        fat = (9.0 / 8.0) * eta * (u + FAT_NOISE * gauss(u.shape, g))
        yield by_parity(fat), by_parity((-1.0 / 24.0) * eta * prod)


def spinors(c, seed, n, parities=1):
    """[n, parities, Vh, 3] Gaussian colour vectors."""
    return gauss((n, parities, volume(c) // 2, 3), generator(seed, 100))


def weights(seed):
    """Weights W[o][i][p] (re, im) of every layer: a dominant identity path and small random mixing."""
    rng = np.random.default_rng(int(seed) + 7)
    out = []
    for ci, co in zip(CHANNELS[:-1], CHANNELS[1:]):
        w = 0.05 * rng.standard_normal((co, ci, 9, 2))
        w[0, 0, 0, 0] += 1.0
        out.append(w.astype(np.float32))
    return out


# ---------------------------------------------------------------------------------------------------- device fields
def planes(f, pv):
    """[..., Vh, 3] complex -> the FP64 device layout (three planes of pv (re, im) pairs) as flat float64."""
    out = torch.zeros(*f.shape[:-2], 3, pv, dtype=torch.complex128, device=f.device)
    out[..., : f.shape[-2]] = f.transpose(-1, -2)
    return torch.view_as_real(out).reshape(-1)


def planes32(f, pv):
    """[..., Vh, 3] complex -> the order of the FP32 device layout (two colours per site, then the third)."""
    out = torch.zeros(*f.shape[:-2], pv, 3, dtype=torch.complex128, device=f.device)
    out[..., : f.shape[-2], :] = f
    r = torch.view_as_real(out)
    a, b = r[..., :2, :].flatten(-3), r[..., 2:, :].flatten(-3)
    return torch.cat([a, b], -1).reshape(-1)


def load(c, seed, prec=64):
    ctx = K.Context(dims_of(c))
    v = volume(c)
    rec = torch.empty(2, v, 4, 9, dtype=torch.complex128, device="cuda")
    for mu, fl in enumerate(links(c, seed)):
        for t in (0, 1):
            rec[t, :, mu] = fl[t].reshape(v, 9)
    del fl
    host = torch.empty(v * 72, dtype=torch.float64, pin_memory=True)
    for t, kind in enumerate((K.KUQCD_FAT_LINK, K.KUQCD_LONG_LINK)):
        host.copy_(torch.view_as_real(rec[t]).reshape(-1))
        ctx.load_links(kind, host.numpy())
    del rec
    torch.cuda.empty_cache()
    for p in {64: (64,), 32: (64, 32), 16: (64, 32, 16)}[prec]:
        ctx.prepare(PREC[p])
    return ctx


def field(ctx, prec, n=1):
    return torch.zeros(ctx.spinor_bytes(PREC[prec]) * n, dtype=torch.uint8, device="cuda")


def put(ctx, f, prec=64, like=None):
    """[..., Vh, 3] complex -> device fields of a precision (bytes)."""
    pv = ctx.spinor_bytes(K.KUQCD_DOUBLE) // 48
    d = planes(f, pv).view(torch.uint8)
    if prec == 64:
        return d
    n = d.numel() // ctx.spinor_bytes(K.KUQCD_DOUBLE)
    out = field(ctx, prec, n)
    a, b = ctx.spinor_bytes(K.KUQCD_DOUBLE), ctx.spinor_bytes(PREC[prec])
    for k in range(n):
        ctx.convert(d[k * a:(k + 1) * a], K.KUQCD_DOUBLE, out[k * b:(k + 1) * b], PREC[prec])
    torch.cuda.synchronize()
    return out


def prepare(c, seed):
    kind = c["kind"]
    s = {"c": c, "sig": sigmas(c)}
    if kind in ("op", "full"):
        p = c["prec"]
        halves = 2 if kind == "full" else 1
        s["ctx"] = ctx = load(c, seed, p)
        s["src"] = put(ctx, spinors(c, seed, 1, halves)[0], 64 if p == 16 else p)
        s["dst"], s["tmp"] = field(ctx, p, halves), field(ctx, p, halves)
        if p == 16:
            s["in16"], s["out32"] = field(ctx, 16), field(ctx, 32)
    elif kind == "solve":
        s["ctx"] = ctx = load(c, seed, 64 if c["solver"] == "cgm" else 16)
        b = spinors(c, seed, 1)[0, 0]
        s["tol"] = RES ** 2 * float(b.abs().square().sum())
        if c["host"]:
            s["b"] = torch.view_as_real(b).reshape(-1).cpu().numpy()
        else:
            s["b"], s["x"] = put(ctx, b), field(ctx, 64, c["shifts"])
    elif kind == "residuals":
        s["ctx"] = ctx = load(c, seed)
        b, x = candidates(c, seed)
        s["b"], s["x"] = put(ctx, b), put(ctx, x)
    elif kind == "batch":
        s["ctx"] = ctx = load(c, seed, 16)
        s["b"] = [put(ctx, b) for b in spinors(c, seed, c["sources"])[:, 0]]
        s["x"] = [field(ctx, 64, c["shifts"]) for _ in s["b"]]
        s["batch"] = K.Batch()
        for b, x in zip(s["b"], s["x"]):
            s["batch"].add(ctx, b, x, s["sig"], solver=K.KQ_SOLVER_MIXED, prec=K.KUQCD_HALF, rel_residual=RES)
    else:
        s["ctx"] = ctx = load(c, seed, 32)
        s["net"] = net = K.Net(ctx, CHANNELS)
        net.weights = np.concatenate([w.ravel() for w in weights(seed)])
        if c["train"]:
            r, e = pair(c, seed)
            s["r"], s["e"], s["e2"] = put(ctx, r), put(ctx, e), float(e.abs().square().sum())
        else:
            s["r"], s["out"] = put(ctx, spinors(c, seed, 1)[0, 0]), field(ctx, 64)
    return s


def run(s):
    c, ctx, kind = s["c"], s["ctx"], s["c"]["kind"]
    if kind == "op":
        p = PREC[c["prec"]]
        if c["prec"] == 16:
            ctx.convert(s["src"], K.KUQCD_DOUBLE, s["in16"], p)
            ctx.mdagm(p, s["sig"][0], s["in16"], s["dst"], s["tmp"], 0)
            ctx.convert(s["dst"], p, s["out32"], K.KUQCD_SINGLE)
            return s["out32"].view(torch.float32)
        ctx.mdagm(p, s["sig"][0], s["src"], s["dst"], s["tmp"], 0)
        return s["dst"].view(torch.float64 if c["prec"] == 64 else torch.float32)
    if kind == "full":
        ctx.mdagm_full(PREC[c["prec"]], s["sig"][0], s["src"], s["dst"], s["tmp"])
        return s["dst"].view(torch.float64 if c["prec"] == 64 else torch.float32)
    if kind == "solve":
        how = (dict(solver=K.KQ_SOLVER_CGM, prec=K.KUQCD_DOUBLE, tol=s["tol"]) if c["solver"] == "cgm" else
               dict(solver=K.KQ_SOLVER_MIXED, prec=K.KUQCD_HALF, rel_residual=RES))
        if c["host"]:
            return ctx.solve(s["b"], s["sig"], **how)[0]
        ctx.solve_device(s["b"], s["x"], s["sig"], **how)
        return s["x"].view(torch.float64)
    if kind == "residuals":
        return np.array(ctx.true_residuals(0, s["sig"], s["b"], s["x"]))
    if kind == "batch":
        s["batch"].solve()
        return [x.view(torch.float64) for x in s["x"]]
    net = s["net"]
    if c["train"]:
        net.zero_grad()
        loss = net.train_pair(s["r"], s["e"], 0, s["e2"])
        return {"loss": loss, "grad": net.grad()}
    net.apply(s["r"], s["out"], 0)
    return s["out"].view(torch.float64)


# ---------------------------------------------------------------------------------------------------- work
def work(c):
    v, vh = volume(c), volume(c) // 2
    kind = c["kind"]
    word = {64: 8, 32: 4, 16: 2}
    spin = {64: 48, 32: 24, 16: 16}
    # one dslash: 16 links and 1146 flops per output site
    link = lambda p: 16 * 18 * word[p]  # noqa: E731
    if kind in ("op", "full"):
        p, n = c["prec"], vh * (2 if kind == "full" else 1)
        # the links, which both halves of the operator share, the source and the result, each once
        links_once = 8 * 2 * vh * 18 * word[p]
        edge = (48 + 24) if p == 16 else 2 * spin[p]
        return {"bytes": links_once + n * edge, "flops": n * (2 * 1146 + 12)}
    if kind == "solve":
        # every iteration applies the operator once (both halves; half of the links' words may be short ones in the
        # mixed solver) and updates the base vectors; every solution is written once
        share = 0.5 if c["solver"] == "mixed" else 1.0
        per = vh * (2 * share * link(64) + 6 * 48)
        return {"bytes": ITERS * per + vh * 48 * (1 + c["shifts"]),
                "flops": ITERS * vh * (2 * 1146 + 12 * (3 + c["shifts"]))}
    if kind == "residuals":
        return {"bytes": 8 * v * 144 + vh * 48 * (1 + c["shifts"]), "flops": c["shifts"] * vh * (2 * 1146 + 36)}
    if kind == "batch":
        n = c["sources"]
        per = vh * (2 * 0.5 * link(64) + n * 6 * 48)
        return {"bytes": ITERS * per + n * vh * 48 * (1 + c["shifts"]),
                "flops": n * ITERS * vh * (2 * 1146 + 12 * (3 + c["shifts"]))}
    # the fat links once per layer, every activation written and read once; transports (8 matrices of 66 flops per
    # channel) and the channel mixing of every layer of M (and, in training, of its weight gradients)
    mid = sum(CHANNELS[1:-1]) * 2 + CHANNELS[-1]
    layers = 2 * (len(CHANNELS) - 1)
    apply_ = v * (layers * 4 * 72 + 2 * 24 * mid) + vh * 96
    flops = sum(2 * v * 3 * (8 * 22 * ci + 8 * 9 * ci * co) for ci, co in zip(CHANNELS[:-1], CHANNELS[1:]))
    return {"bytes": apply_ * (3 if c["train"] else 1), "flops": flops * (3 if c["train"] else 1)}


# ---------------------------------------------------------------------------------------------------- 64-bit values
class Operator:
    """The hopping term on gathered neighbours, factors 1/2 (fat) and -1/48 (long) included."""

    def __init__(self, c, seed, fat_only=False):
        self.dims = nx, ny, nz, nt = dims_of(c)
        self.vh = volume(c) // 2
        i = torch.arange(self.vh, device="cuda")
        hx = nx // 2
        xcb, r = i % hx, i // hx
        pos = [None, r % ny, r // ny % nz, r // ny // nz]
        self.nbr, self.terms = {}, {0: [], 1: []}
        stride = [0, hx, hx * ny, hx * ny * nz]
        for p in (0, 1):
            x = 2 * xcb + (pos[1] + pos[2] + pos[3] + p) % 2
            for mu in range(4):
                for hop in (1, -1, 3, -3):
                    if mu == 0:
                        j = i - xcb + (x + hop) % nx // 2
                    else:
                        j = i + ((pos[mu] + hop) % self.dims[mu] - pos[mu]) * stride[mu]
                    self.nbr[p, mu, hop] = j
        for mu, (fat, lng) in enumerate(links(c, seed)):
            for hop, f, w in ((1, fat, 0.5), (3, lng, -1.0 / 48.0)):
                if fat_only and hop == 3:
                    continue
                f = w * f
                for p in (0, 1):
                    back = f[1 - p][self.nbr[p, mu, -hop]].mH.contiguous()
                    self.terms[p].append((f[p].contiguous(), self.nbr[p, mu, hop], 1.0))
                    self.terms[p].append((back, self.nbr[p, mu, -hop], -1.0))

    def dslash(self, v, p):
        """[..., Vh, 3] of parity 1 - p -> parity p."""
        out = torch.zeros_like(v)
        for u, j, sign in self.terms[p]:
            w = v[..., j, :]
            for k in range(3):
                out.addcmul_(u[..., :, k], w[..., k, None], value=sign)
        return out

    def apply(self, sigma, v, p=0):
        return sigma * v - self.dslash(self.dslash(v, 1 - p), p)


def multishift(op, b, sig, tol=1e-13):
    """Multishift CG (recurrences of the shifted systems) with FP64 vectors and scalars."""
    ns = len(sig)
    x = torch.zeros(ns, *b.shape, dtype=b.dtype, device=b.device)
    p = b.expand(ns, *b.shape).clone()
    r, rr = b.clone(), float(b.abs().square().sum())
    stop = tol * tol * rr
    z, zo, al_o, be = np.ones(ns), np.ones(ns), 1.0, 0.0
    d = np.array(sig) - sig[0]
    for _ in range(5000):
        q = op.apply(sig[0], p[0])
        al = rr / float((p[0].conj() * q).real.sum())
        ns = int((np.abs(z) > 1e-30).sum())  # the largest shifts are done long before the smallest
        z, zo = z[:ns], zo[:ns]
        zn = z * zo * al_o / (al * be * (zo - z) + zo * al_o * (1.0 + d[:ns] * al))
        x[:ns] += torch.from_numpy(al * zn / z).to(b.device).reshape(ns, 1, 1) * p[:ns]
        r = r - al * q
        new = float(r.abs().square().sum())
        be_new = new / rr
        bk = torch.from_numpy(be_new * (zn / z) ** 2).to(b.device).reshape(ns, 1, 1)
        p[:ns] *= bk
        p[:ns] += torch.from_numpy(zn).to(b.device).reshape(ns, 1, 1) * r
        zo, z, al_o, be, rr = z, zn, al, be_new, new
        if rr < stop:
            return x
    return None


def candidates(c, seed):
    """A source and, for every shift, a first approximation of its solution."""
    b = spinors(c, seed, 1)[0, 0]
    return b, torch.stack([b / (s + 2.0) for s in sigmas(c)])


def pair(c, seed):
    """A training pair as a solver leaves it: an error e and its residual r = A e."""
    e = spinors(c, seed, 1)[0, 0]
    return Operator(c, seed).apply(MASS2 + SMIN, e), e


def network(op, ws, v):
    """M v = P^T N^dag N P v on the full lattice; ws: per layer complex [o, i, 9]."""
    hop = {p: [(u, j, sign) for u, j, sign in op.terms[p]] for p in (0, 1)}

    def transport(a, path):  # a: [channels, 2, Vh, 3]
        if path == 0:
            return a
        out = []
        for p in (0, 1):
            u, j, _ = hop[p][path - 1]
            out.append((u * a[:, 1 - p][:, j][..., None, :]).sum(-1))
        return torch.stack(out, 1)

    swap = [0, 2, 1, 4, 3, 6, 5, 8, 7]
    a = torch.stack([v, torch.zeros_like(v)])[None]
    for w in ws:
        a = sum(torch.einsum("oi,ipvc->opvc", w[:, :, k], transport(a, k)) for k in range(9))
    for w in reversed(ws):
        a = sum(torch.einsum("oi,opvc->ipvc", w[:, :, k].conj(), transport(a, swap[k])) for k in range(9))
    return a[0, 0]


def exact(c, seed):
    kind, v = c["kind"], volume(c)
    pv = (v // 2 + 63) // 64 * 64
    if kind in ("op", "full"):
        halves = 2 if kind == "full" else 1
        src = spinors(c, seed, 1, halves)[0]
        if v > 4_000_000:
            return None
        op, sig = Operator(c, seed), sigmas(c)[0]
        out = torch.stack([op.apply(sig, src[p], p) for p in range(halves)])
        return planes(out, pv) if c["prec"] == 64 else planes32(out, pv)
    if kind == "solve":
        b = spinors(c, seed, 1)[0, 0]
        x = multishift(Operator(c, seed), b, sigmas(c))
        if x is None:
            return None
        return [torch.view_as_real(k).reshape(-1) for k in x] if c["host"] else planes(x, pv)
    if kind == "residuals":
        op, (b, x) = Operator(c, seed), candidates(c, seed)
        off = [(b - op.apply(s, xk)).abs().square().sum() for s, xk in zip(sigmas(c), x)]
        return torch.stack([(o / b.abs().square().sum()).sqrt() for o in off])
    if kind == "batch":
        op = Operator(c, seed)
        xs = [multishift(op, b, sigmas(c)) for b in spinors(c, seed, c["sources"])[:, 0]]
        return None if any(x is None for x in xs) else [planes(x, pv) for x in xs]
    op = Operator(c, seed, fat_only=True)
    # the transports use F and F^dag without the hopping term's sign
    ws = [torch.from_numpy(w).double().cuda().requires_grad_(c["train"]) for w in weights(seed)]
    cw = [torch.view_as_complex(w) for w in ws]
    if not c["train"]:
        with torch.no_grad():
            return planes(network(op, cw, spinors(c, seed, 1)[0, 0]), pv)
    r, e = pair(c, seed)
    loss = (network(op, cw, r) - e).abs().square().sum() / e.abs().square().sum()
    loss.backward()
    return {"loss": loss.detach(), "grad": torch.cat([w.grad.reshape(-1) for w in ws])}
