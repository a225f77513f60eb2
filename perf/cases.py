"""The solver's work as its users call it, for measuring.

Every case is one call sequence through the public Python API on one lattice:
single operators, the SAP preconditioners (the layer the solvers spend their
time in), the even-odd family, the clover term a request with a new kappa
needs, and two whole solves.  Lattices are written "XxYxZxT", block grids
"a.b.c.d"; gauge fields are SU(3) after 5 APE steps with csw = 1.7, the
fields of this repository's own benchmark.

`exact` restates the field generator and every operator in torch, in FP64 and
in natural site order, and lays the result out in the device planes of the
public ABI (include/qwsg.h).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qws_b200

CSW = 1.7
_stream = None


def _case(name, kind, L, NB="2.1.1.1", kappa=0.1365, nsap=4, nm=2, nrhs=1):
    c = dict(kind=kind, L=L, NB=NB, kappa=kappa, nsap=nsap, nm=nm, nrhs=nrhs)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the FP64 operator of the outer residual, at a production volume
        _case("dslash_f64_24c48", "dslash_f64", "24x24x24x48"),
        # the FP32 operator on a ragged lattice: odd block extents, sites that
        # do not fill the planes' padding
        _case("dslash_f32_ragged", "dslash_f32", "20x14x6x18", "4.2.2.2"),
        # the plain solver's preconditioner (D M_SAP) on the headline lattice,
        # at the reference's partition: one inner half-iteration
        _case("sap_f32_32c64", "sap_f32", "32x32x32x64"),
        # the same on the smallest lattice the service takes: latency
        _case("sap_f32_8c8", "sap_f32", "8x8x8x8", "2.2.2.2"),
        # the precision form's FP16-storage preconditioner in its tuned
        # partition on the headline lattice
        _case("sap_f16_32c64", "sap_f16", "32x32x32x64", "2.2.2.2", nm=3),
        # many right-hand sides of one gauge field (the batch of spin-colour sources)
        _case("sap_f16_24c48_rhs8", "sap_f16", "24x24x24x48", "2.2.2.2", nm=3, nrhs=8),
        # a merged batch of requests, each with its own kappa: clover terms
        # built on the device, then one preconditioner application
        _case("request_batch_16c32", "kappas", "16x16x16x32", "2.2.2.2", nm=3, nrhs=4),
        # one request with a new kappa: the clover term and the FP64 and FP32
        # operators with it
        _case("request_kappa_24c48", "clover", "24x24x24x48", "2.2.2.2", kappa=0.1340),
        # the even-odd normal operator in FP64 (the HMC's force solves), alone
        _case("evenodd_f64_24c48", "eo_f64", "24x24x24x48"),
        # ... and as CG to its 1e-14
        _case("evenodd_cg_16c32", "cg", "16x16x16x32", kappa=0.1300),
        # the plain solve to 1e-10, reference partition
        _case("solve_plain_16c32", "solve", "16x16x16x32"),
        # the precision form's solve to 1e-10, tuned partition
        _case("solve_precision_24c48", "solve_hf", "24x24x24x48", "2.2.2.2", nm=3),
    ]


#: drawn kinds with the largest volume each is drawn up to
_DRAW = [("dslash_f64", 1 << 21), ("dslash_f32", 1 << 21), ("sap_f32", 1 << 20), ("sap_f16", 1 << 20),
         ("sap_f16_rhs", 1 << 17), ("kappas", 1 << 16), ("clover", 1 << 18), ("eo_f64", 1 << 20),
         ("eo_f32", 1 << 20), ("cg", 1 << 16), ("solve", 1 << 17), ("solve_hf", 1 << 18)]


def draw(rng):
    kind, most = rng.choice(_DRAW)
    while True:
        # even extents 4 .. 40 (odd block extents come with them), a volume
        # spread over the logarithm of the range, kappa of the serving mix
        want = math.exp(rng.uniform(math.log(4096), math.log(most)))
        side = want ** 0.25
        L = [2 * max(2, min(20, round(side * rng.uniform(0.55, 1.8) / 2))) for _ in range(4)]
        if 0.8 * want < math.prod(L) < min(most, 1.25 * want):
            break
    NB = [2] + [rng.choice((1, 2)) for _ in range(3)]
    if L[0] % 4 == 0 and L[0] > 12 and rng.random() < 0.3:
        NB[0] = 4
    nrhs = 1
    if kind == "sap_f16_rhs":
        kind, nrhs = "sap_f16", rng.choice((2, 4, 8, 16))
    if kind == "kappas":
        nrhs = rng.choice((2, 4, 8))
    kappa = round(rng.uniform(0.1300, 0.1345 if kind == "cg" else 0.1365), 5)
    return _case(None, kind, "x".join(map(str, L)), ".".join(map(str, NB)), kappa,
                 rng.choice((3, 4)), rng.choice((2, 3)), nrhs)


def _dims(case):
    return [int(v) for v in case["L"].split("x")], [int(v) for v in case["NB"].split(".")]


def _kappas(case):
    """a kappa per right-hand side, downwards from the case's own"""
    return [case["kappa"] - 0.0007 * r for r in range(case["nrhs"])]


def _source(case, seed):
    """Gaussian sources [nrhs, V, 24] in natural order, FP64 on the host"""
    L, _ = _dims(case)
    g = torch.Generator(device="cpu").manual_seed(1000003 * seed + 17)
    return torch.randn((case["nrhs"], math.prod(L), 24), generator=g, dtype=torch.float32).double()


_FP64 = ("dslash_f64", "clover", "eo_f64", "cg", "solve", "solve_hf")


def prepare(case, seed):
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()  # (graphs are off on the default stream)
    L, NB = _dims(case)
    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=case["kappa"], stream=_stream)
    lat.gen_gauge_device(seed, 5, 0.36)
    lat.build_clover(CSW)
    one = lat if case["nrhs"] == 1 else lat.batch(case["nrhs"], stream=_stream)
    b = _source(case, seed).numpy()
    b = b[0] if case["nrhs"] == 1 else b
    s = dict(case=case, lat=lat, one=one)
    f64 = case["kind"] in _FP64
    s["b"] = one.to_device(b if f64 else b.astype(np.float32))
    s["out"] = one.empty("f64" if f64 else "f32")
    if case["kind"] == "clover":
        s["b32"] = lat.to_device(b.astype(np.float32))
        s["out32"] = lat.empty("f32")
    if case["kind"] == "cg":
        s["maxiter"] = 2000
    torch.cuda.synchronize()
    return s


def run(s):
    case, lat, one, b, out = s["case"], s["lat"], s["one"], s["b"], s["out"]
    kind, nsap, nm = case["kind"], case["nsap"], case["nm"]
    if kind in ("dslash_f64", "dslash_f32"):
        return one.ddd(b, out=out)
    if kind == "sap_f32":
        return one.prec_ddd(b, nsap, nm, out=out)
    if kind == "sap_f16":
        return one.prec_h(b, nsap, nm, out=out)
    if kind == "kappas":
        one.set_kappas(_kappas(case), CSW)
        return one.prec_h(b, nsap, nm, out=out)
    if kind == "clover":
        lat.set_kappa(case["kappa"])
        lat.build_clover(CSW)
        return [one.ddd(b, out=out), one.ddd(s["b32"], out=s["out32"])]
    if kind == "eo_f64":
        return one.mtdagmt(b, out=out)
    if kind == "eo_f32":
        return one.mtilde(b, out=out)
    with torch.cuda.stream(_stream):
        out.zero_()  # the initial guess
    if kind == "cg":
        one.cg_vm(out, b, s["maxiter"])
    elif kind == "solve":
        one.bicgstab_dd_mix(out, b, 1e-10, 100, 1e-6, 50, nsap, nm)
    else:
        one.bicgstab_dd_mix2_hf(out, b, 1e-10, 100, 1e-6, 50, nsap, nm, reliable=5)
    return out


def _operators(case):
    """applications of D, or of D on one colour as a half, that one pass needs"""
    kind, nsap, nm = case["kind"], case["nsap"], case["nm"]
    sap = lambda sweeps: sweeps * (nm + 1) + nm
    n = {"dslash_f64": 1, "dslash_f32": 1, "sap_f32": sap(nsap) + 1, "sap_f16": sap(nsap - 1),
         "kappas": sap(nsap - 1), "clover": 2, "eo_f64": 2, "eo_f32": 1}
    # solves: about that many operator applications on these fields
    n.update(cg=2 * 250, solve=30 * (sap(nsap) + 1), solve_hf=30 * (sap(nsap - 1) + 1))
    return n[kind]


def work(case):
    L, _ = _dims(case)
    V, n, kind = math.prod(L), case["nrhs"], case["kind"]
    real = 8 if kind in _FP64 else 4
    fields = real * 72 * 2  # links and inverse clover of a site
    if kind in ("kappas", "sap_f16") and n > 1:
        fields = real * 72 * (1 + (n if kind == "kappas" else 1))
    bytes_ = V * (2 * 24 * real * n + fields)
    flops = V * 1872 * _operators(case) * n
    if kind in ("clover", "kappas"):
        # the clover term is made here, not read: four leaves on six planes, two 6x6 inverses
        bytes_ = V * (72 * 8 + 2 * 24 * real * n + (2 * 24 * 4 if kind == "clover" else 0))
        flops += V * (24 * 3 * 198 + 2 * 2000 * n)
    if kind in ("eo_f64", "eo_f32", "cg"):  # one parity in and out
        bytes_ = V * (24 * real + fields)
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    """About four times the distance from `exact` that the operators showed, or,
    for a solve, what its stopping rule leaves open."""
    kind = case["kind"]
    if kind in ("dslash_f64", "eo_f64"):
        return {"rel": 4e-15, "max": 2e-13}
    if kind in ("dslash_f32", "eo_f32", "clover"):
        return {"rel": 4e-7, "max": 2e-5}
    if kind == "sap_f32":
        return {"rel": 1e-6, "max": 5e-5}
    if kind in ("sap_f16", "kappas"):
        return {"rel": 2e-3, "max": 0.05}
    if kind == "cg":
        return {"rel": 1e-12, "max": 5e-11}
    return {"rel": 1e-9, "max": 1e-7}  # a solve to a residual of 1e-10


# ---------------------------------------------------------------------------
# the same in FP64, without this repository's code
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _shr(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


def _splitmix(x):
    x = x + _i64(0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _i64(0xBF58476D1CE4E5B9)
    x = (x ^ _shr(x, 27)) * _i64(0x94D049BB133111EB)
    return x ^ _shr(x, 31)


def _su3(m):
    """Gram-Schmidt on the rows, then the determinant phase divided out"""
    rows = []
    for i in range(3):
        r = m[..., i, :]
        for q in rows:
            r = r - (q.conj() * r).sum(-1, keepdim=True) * q
        rows.append(r / r.abs().square().sum(-1, keepdim=True).sqrt())
    a, b, c = rows
    d = (a * torch.linalg.cross(b, c)).sum(-1)
    ph = torch.polar(torch.ones_like(d.real), -d.angle() / 3)
    return torch.stack(rows, -2) * ph[..., None, None]


class _Exact:
    """One lattice in FP64: fields are [T, Z, Y, X, ...]"""

    #: spin part of 1 + G for a forward hop (1 - G backward): rows (column, factor)
    G = [[(3, -1j), (2, -1j), (1, 1j), (0, 1j)], [(3, -1), (2, 1), (1, 1), (0, -1)],
         [(2, -1j), (3, 1j), (0, 1j), (1, -1j)], [(0, -1), (1, -1), (2, 1), (3, 1)]]

    def __init__(self, case, seed):
        self.L, self.NB = _dims(case)
        self.B = [l // n for l, n in zip(self.L, self.NB)]
        self.kappa = case["kappa"]
        self.dev = _dev()
        X, Y, Z, T = self.L
        ax = [torch.arange(n, device=self.dev) for n in (T, Z, Y, X)]
        t, z, y, x = torch.meshgrid(*ax, indexing="ij")
        self.x = [x, y, z, t]
        bc = [c // b for c, b in zip(self.x, self.B)]
        self.colour = sum(bc) % 2
        self.parity = (x + y + z + t) % 2
        self.U = self._gauge(seed)
        self.F = self._leaves()
        self.set_kappa(self.kappa)

    def shift(self, f, mu, d):
        """f(x + d mu)"""
        return torch.roll(f, -d, 3 - mu)

    def _gauge(self, seed):
        n = self.x[0] + self.L[0] * (self.x[1] + self.L[1] * (self.x[2] + self.L[2] * self.x[3]))
        U = []
        for mu in range(4):
            key = n * 0x100000001B3 + _i64(mu * 0x9E3779B97F4A7C15)
            state = _splitmix(_splitmix(key) ^ seed)
            m = []
            for _ in range(9):
                u = []
                for _ in range(2):
                    state = state + _i64(0x9E3779B97F4A7C15)
                    u.append((_shr(_splitmix(state), 11) + 1).double() / 9007199254740992.0)
                m.append(torch.polar((-u[0].log()).sqrt(), 2 * math.pi * u[1]))
            U.append(_su3(torch.stack(m, -1).reshape(*n.shape, 3, 3)))
        for _ in range(5):
            W = []
            for mu in range(4):
                S = 0
                for nu in range(4):
                    if nu == mu:
                        continue
                    S = S + U[nu] @ self.shift(U[mu], nu, 1) @ self.shift(U[nu], mu, 1).mH
                    S = S + self.shift(U[nu].mH @ U[mu] @ self.shift(U[nu], mu, 1), nu, -1)
                W.append(_su3((1 - 0.36) * U[mu] + 0.36 / 6 * S))
            U = W
        return U

    def _leaves(self):
        """F_{mu nu} = (Q - Q^dag) / (8i), traceless, Q the four-leaf sum"""
        F = {}
        s, U = self.shift, self.U
        for m in range(4):
            for n in range(m + 1, 4):
                P = U[m] @ s(U[n], m, 1) @ s(U[m], n, 1).mH @ U[n].mH
                Q = P
                Q = Q + U[n] @ s(s(U[m], n, 1), m, -1).mH @ s(U[n], m, -1).mH @ s(U[m], m, -1)
                Q = Q + (s(U[m], m, -1).mH @ s(s(U[n], m, -1), n, -1).mH
                         @ s(s(U[m], m, -1), n, -1) @ s(U[n], n, -1))
                Q = Q + s(U[n], n, -1).mH @ s(U[m], n, -1) @ s(s(U[n], n, -1), m, 1) @ U[m].mH
                f = (Q - Q.mH) / 8j
                tr = f.diagonal(dim1=-2, dim2=-1).sum(-1) / 3
                F[m, n] = f - tr[..., None, None] * torch.eye(3, device=self.dev)
        return F

    def set_kappa(self, kappa):
        """the inverse of T = 1 - csw kappa sum sigma F, as two 6x6 blocks (spins s0 +- s2, s1 +- s3)"""
        self.kappa = kappa
        gam = np.zeros((4, 4, 4), complex)
        for mu in range(4):
            for r, (col, f) in enumerate(self.G[mu]):
                gam[mu, r, col] = -f
        P = np.array([[1, 0, 1, 0], [0, 1, 0, 1], [1, 0, -1, 0], [0, 1, 0, -1]])
        self.inv = []
        for blk in range(2):
            T = torch.eye(6, dtype=torch.complex128, device=self.dev).expand(*self.x[0].shape, 6, 6)
            T = T.clone().unflatten(-2, (2, 3)).unflatten(-1, (2, 3))
            for (m, n), f in self.F.items():
                sig = 0.5j * (gam[m] @ gam[n] - gam[n] @ gam[m])
                S = (P @ sig @ P.T / 2)[2 * blk:2 * blk + 2, 2 * blk:2 * blk + 2]
                for h in range(2):
                    for k in range(2):
                        if S[h, k] != 0:
                            T[..., h, :, k, :] -= CSW * kappa * complex(S[h, k]) * f
            self.inv.append(torch.linalg.inv(T.flatten(-4, -3).flatten(-2, -1)))

    def clover(self, v):
        """A^-1 v; v [..., 3 colours, 4 spins]"""
        s0, s1, s2, s3 = v.unbind(-1)
        x = [torch.cat((s0 + s2, s1 + s3), -1), torch.cat((s0 - s2, s1 - s3), -1)]
        y = [(self.inv[i] @ x[i][..., None])[..., 0] / 2 for i in range(2)]
        p, q = y[0] + y[1], y[0] - y[1]
        return torch.stack((p[..., :3], p[..., 3:], q[..., :3], q[..., 3:]), -1)

    def _proj(self, v, mu, sign):
        cols = [c for c, _ in self.G[mu]]
        f = torch.tensor([complex(f) for _, f in self.G[mu]], dtype=torch.complex128, device=self.dev)
        return v + sign * v[..., cols] * f

    def hops(self, v, which="all", dag=1):
        """sum of the hops; which: all, inner (stay in their block) or outer"""
        out = torch.zeros_like(v)
        for mu in range(4):
            lc = self.x[mu] % self.B[mu]
            for d in (1, -1):
                face = lc == (self.B[mu] - 1 if d > 0 else 0)
                h = self._proj(v, mu, d * dag)
                if d > 0:
                    h = self.U[mu] @ self.shift(h, mu, 1)
                else:
                    h = self.shift(self.U[mu].mH @ h, mu, -1)
                if mu == 3:  # antiperiodic in time
                    edge = self.x[3] == (self.L[3] - 1 if d > 0 else 0)
                    h = torch.where(edge[..., None, None], -h, h)
                if which != "all":
                    keep = face if which == "outer" else ~face
                    h = h * keep[..., None, None]
                out += h
        return out

    def D(self, v):
        return v - self.kappa * self.clover(self.hops(v))

    def on(self, mask, a, b):
        return torch.where(mask[..., None, None], a, b)

    def jinv(self, s, nm):
        x = s
        for _ in range(max(1, nm)):
            x = s + self.kappa * self.clover(self.hops(x, "inner"))
        return x

    def sap(self, b, sweeps, nm):
        k = self.kappa
        s, a = b.clone(), torch.zeros_like(b)
        for _ in range(sweeps):
            for e in range(2):
                mine = self.colour == e
                se = self.on(mine, s, torch.zeros_like(s))
                a = self.on(mine, self.jinv(se, nm), a)
                ae = self.on(mine, a, torch.zeros_like(a))
                s = self.on(mine, s + b - (ae - k * self.clover(self.hops(ae, "inner"))), s)
                s = self.on(~mine, s + k * self.clover(self.hops(a, "outer")), s)
        even = self.colour == 0
        zero = torch.zeros_like(s)
        xe = self.on(even, self.jinv(self.on(even, s, zero), nm), zero)
        s = self.on(~even, s + k * self.clover(self.hops(xe, "outer")), s)
        return self.on(even, xe, self.jinv(self.on(even, zero, s), nm))

    def schur(self, v, dag=False):
        """even sites: 1 - kappa^2 A^-1 H A^-1 H (mtilde) or its adjoint"""
        even = self.parity == 0
        zero = torch.zeros_like(v)
        v = self.on(even, v, zero)
        if not dag:
            w = self.clover(self.hops(self.on(even, zero, self.clover(self.hops(v)))))
        else:
            w = self.hops(self.on(even, zero, self.clover(self.hops(self.clover(v), dag=-1))), dag=-1)
        return self.on(even, v - self.kappa ** 2 * w, zero)

    def solve(self, A, b, tol):
        """BiCGStab"""
        dot = lambda p, q: torch.vdot(p.flatten(), q.flatten())
        x = torch.zeros_like(b)
        r = b.clone()
        r0, p = r.clone(), r.clone()
        rho = dot(r0, r)
        bb = b.norm()
        for _ in range(2000):
            q = A(p)
            alpha = rho / dot(r0, q)
            s = r - alpha * q
            t = A(s)
            om = dot(t, s) / dot(t, t)
            x = x + alpha * p + om * s
            r = s - om * t
            if r.norm() < tol * bb:
                break
            rho1 = dot(r0, r)
            p = r + (rho1 / rho) * (alpha / om) * (p - om * q)
            rho = rho1
        return x

    # ---- natural arrays <-> fields, and the device planes --------------------
    def field(self, nat):
        X, Y, Z, T = self.L
        v = torch.view_as_complex(nat.reshape(T, Z, Y, X, 3, 4, 2).contiguous().to(self.dev))
        return v

    def site_order(self):
        """DD order: colour, block, then the block's directions from slowest to fastest"""
        B, NB, x = self.B, self.NB, self.x
        d = sorted((3, 2, 1, 0), key=lambda m: -B[m])
        order = [d[1], d[2], d[3], d[0]]
        for f in range(4):
            slow = d[1 if f == 0 else 0]
            if math.prod(B) // B[slow] <= 16384:
                order = [d[f]] + [m for m in d if m != d[f] and m != slow] + [slow]
                break
        bc = [c // b for c, b in zip(x, B)]
        local, stride = 0, 1
        for k, m in enumerate(order):
            l = x[m] % B[m]
            if k == 0:  # the fastest row is stored rotated by one
                l = (l + 1) % B[m]
            local = local + l * stride
            stride *= B[m]
        lin = bc[0] + NB[0] * (bc[1] + NB[1] * (bc[2] + NB[2] * bc[3]))
        return self.colour * (math.prod(self.L) // 2) + (lin // 2) * stride + local

    def planes(self, fields, width):
        """FP64 fields of the RHS -> the planes of `width` reals per site and RHS"""
        V = math.prod(self.L)
        pad = (V + 127) // 128 * 128
        out = torch.zeros((24 // width, pad, len(fields), width), dtype=torch.float64, device=self.dev)
        g = self.site_order().flatten()
        for r, f in enumerate(fields):
            out[:, g, r, :] = torch.view_as_real(f).reshape(V, 24 // width, width).transpose(0, 1)
        return out.flatten()


def exact(case, seed):
    kind, nsap, nm = case["kind"], case["nsap"], case["nm"]
    e = _Exact(case, seed)
    src = _source(case, seed)
    b = [e.field(v) for v in src]
    w = 2 if kind in _FP64 else 4
    if kind in ("dslash_f64", "dslash_f32"):
        return e.planes([e.D(b[0])], w)
    if kind == "sap_f32":
        return e.planes([e.D(e.sap(b[0], nsap, nm))], w)
    if kind == "sap_f16":
        return e.planes([e.sap(v, nsap - 1, nm) for v in b], w)
    if kind == "kappas":
        got = []
        for k, v in zip(_kappas(case), b):
            e.set_kappa(k)
            got.append(e.sap(v, nsap - 1, nm))
        return e.planes(got, w)
    if kind == "clover":
        y = e.D(b[0])
        return [e.planes([y], 2), e.planes([y], 4)]
    if kind == "eo_f64":
        return e.planes([e.schur(e.schur(b[0]), dag=True)], w)
    if kind == "eo_f32":
        return e.planes([e.schur(b[0])], w)
    if kind == "cg":
        even = e.on(e.parity == 0, b[0], torch.zeros_like(b[0]))
        y = e.solve(lambda v: e.schur(v, dag=True), even, 1e-14)
        return e.planes([e.solve(e.schur, y, 1e-14)], w)
    return e.planes([e.solve(e.D, b[0], 1e-13)], w)
