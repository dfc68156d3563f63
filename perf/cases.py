"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the public entry points (demo_matrixfree_csem_gb300: Grid, Ctx,
solve_batch, and the device-pointer calls of include/csem_gpu.h):

  dot     csem_cdot_dev          <a, b> for many systems
  A       csem_fdfd_apply_dev    the curl-curl operator, airwave boundary included
  lusgs   csem_lusgs_apply_dev   the LU-SGS preconditioner
  aphi    csem_aphi_apply_dev    the A-phi preconditioner
  solve64 Ctx.solve_fp64         the complex128 drop-in solver, one system, host buffers
  mixed   solve_batch            the batched mixed-precision solver, receivers out

A model is a seeded layered earth under water (or land) on nx x ny x nz core cells, padded
by nb stretched cells per side, as the builders of synthetic.py make them. Vectors look
like Krylov vectors of a dipole source: random, decaying away from the middle of the model.
"""
import ctypes as C
import math

import numpy as np
import torch

import demo_matrixfree_csem_gb300 as cs
from demo_matrixfree_csem_gb300 import api

FREQS = (0.125, 0.25, 0.5, 0.75, 1.0, 1.25)
#: the Marlim-shaped bench model, the 120^3 layered model and the 64^3 one, in core cells
WAVE = dict(nx=180, ny=120, nz=120, hx=200.0, hy=100.0, hz=100.0, nb=10, lextend=120e3, airbc=1, fvm=0, nfft=1024, land=0)
LAYERED120 = dict(nx=100, ny=100, nz=100, hx=100.0, hy=100.0, hz=100.0, nb=10, lextend=40e3, airbc=1, fvm=0, nfft=1024, land=0)
LAYERED64 = dict(nx=64, ny=64, nz=64, hx=100.0, hy=100.0, hz=100.0, nb=10, lextend=40e3, airbc=1, fvm=0, nfft=1024, land=0)
RAGGED = dict(nx=109, ny=93, nz=77, hx=100.0, hy=150.0, hz=50.0, nb=8, lextend=40e3, airbc=0, fvm=1, nfft=1024, land=0)
SMALL_ODD = dict(nx=61, ny=53, nz=47, hx=100.0, hy=100.0, hz=100.0, nb=10, lextend=40e3, airbc=1, fvm=0, nfft=1024, land=0)
TINY = dict(nx=6, ny=5, nz=5, hx=200.0, hy=200.0, hz=100.0, nb=2, lextend=4e3, airbc=1, fvm=0, nfft=256, land=0)


def listed():
    return [
        # the smallest call there is: one dot product of a test-sized system, all latency
        dict(name="dot_c128_small", kind="dot", prec=64, n=2667, nsys=1),
        # the dot products of one wave of the 96-system batch (48 systems of the bench model)
        dict(name="dot_c64_wave48", kind="dot", prec=32, n=11064870, nsys=48),
        # the operator as the batched solver's inner iterations apply it, two frequencies
        dict(name="A_c64_wave16", kind="A", prec=32, nsys=16, nfreq=2, **WAVE),
        # the complex128 operator of the drop-in on an odd-sized finite-volume grid, no airwave
        dict(name="A_c128_ragged", kind="A", prec=64, nsys=1, nfreq=1, **RAGGED),
        # the preconditioner as the batched solver applies it: the largest part of a batch
        dict(name="lusgs_c64_wave16", kind="lusgs", prec=32, nsys=16, nfreq=2, **WAVE),
        # the end of a batch, or a few systems of a small survey: too little work for the chip
        dict(name="lusgs_c64_few", kind="lusgs", prec=32, nsys=3, nfreq=3, **SMALL_ODD),
        # the complex128 preconditioner of the drop-in on the layered 120^3 model
        dict(name="lusgs_c128_layered120", kind="lusgs", prec=64, nsys=1, nfreq=1, **LAYERED120),
        # the other preconditioner (preco=3), on a model without sea water, where it is bounded
        dict(name="aphi_c128_land64", kind="aphi", prec=64, nsys=1, nfreq=1, **dict(LAYERED64, land=1)),
        # a whole drop-in solve of a test-sized model: latency of every launch and status read
        dict(name="solve64_tiny", kind="solve64", algopt=1, preco=1, niter=200, freq=1.0, **TINY),
        # the drop-in solver on the layered 120^3 model, the first iterations of a solve
        dict(name="solve64_layered120", kind="solve64", algopt=1, preco=1, niter=5, freq=0.75, **LAYERED120),
        # a whole batched solve to convergence: six systems on the 64^3 model
        dict(name="mixed_layered64", kind="mixed", algopt=1, niter=1000, max_outer=30, nsys=6, nfreq=2, flow=0.75, **LAYERED64),
        # the batched solver on the bench model, half a wave, the first iterations of a solve
        dict(name="mixed_wave24", kind="mixed", algopt=1, niter=4, max_outer=1, nsys=24, nfreq=3, flow=0.25, **WAVE),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, most, top=(180, 120, 120)):
    """Core cells, spacings and padding; at most `most` unknowns' worth of padded cells."""
    while True:
        n = [_log(rng, 6, t) for t in top]
        nb = rng.choice((4, 8, 10, 15)) if min(n) > 20 else rng.choice((2, 4, 5))
        if (n[0] + 2 * nb) * (n[1] + 2 * nb) * (n[2] + 2 * nb) * 3 <= most:
            break
    return dict(nx=n[0], ny=n[1], nz=n[2], hx=rng.choice((50.0, 100.0, 200.0)), hy=rng.choice((50.0, 100.0, 150.0)),
                hz=rng.choice((50.0, 100.0)), nb=nb, lextend=4e3 if min(n) <= 20 else rng.choice((40e3, 120e3)),
                nfft=1024 if min(n) > 20 else 256)


def draw(rng):
    kind = rng.choice(("dot", "A", "A", "lusgs", "lusgs", "lusgs", "aphi", "solve64", "mixed", "mixed"))
    if kind == "dot":
        n, nsys = _log(rng, 1000, 11000000), _log(rng, 1, 48)
        return dict(kind=kind, prec=rng.choice((32, 64)), n=n, nsys=max(1, min(nsys, 400000000 // n)))
    if kind in ("A", "lusgs"):
        prec = rng.choice((32, 32, 64))
        g = _sizes(rng, 12e6 if prec == 32 else 5.5e6)
        cells = (g["nx"] + 2 * g["nb"]) * (g["ny"] + 2 * g["nb"]) * (g["nz"] + 2 * g["nb"]) * 3
        nsys = max(1, min(_log(rng, 1, 16), int((190e6 if prec == 32 else 5.5e6) / cells)))
        return dict(kind=kind, prec=prec, nsys=nsys, nfreq=rng.randint(1, min(3, nsys)), airbc=rng.choice((0, 1, 1)),
                    fvm=rng.choice((0, 0, 1)), land=0, **g)
    if kind == "aphi":
        g = _sizes(rng, 1.8e6, (64, 64, 64))
        return dict(kind=kind, prec=rng.choice((32, 64)), nsys=rng.randint(1, 2), nfreq=1, airbc=rng.choice((0, 1)),
                    fvm=rng.choice((0, 0, 1)), land=1, **g)
    if kind == "solve64":
        g = _sizes(rng, 5.5e6, (100, 100, 100))
        algopt = rng.choice((1, 1, 2))
        return dict(kind=kind, algopt=algopt, preco=1, niter=10 if algopt == 2 else rng.randint(2, 5),
                    freq=rng.choice(FREQS[1:]), airbc=rng.choice((0, 1)), fvm=0, land=0, **g)
    g = _sizes(rng, 12e6)
    cells = (g["nx"] + 2 * g["nb"]) * (g["ny"] + 2 * g["nb"]) * (g["nz"] + 2 * g["nb"]) * 3
    nsys = max(1, min(_log(rng, 1, 24), int(280e6 / cells)))
    algopt = rng.choice((1, 1, 2))
    return dict(kind=kind, algopt=algopt, niter=5 if algopt == 2 else 4, max_outer=1, nsys=nsys,
                nfreq=rng.randint(1, min(3, nsys)), flow=rng.choice((0.25, 0.5, 0.75)), airbc=1, fvm=0, land=0, **g)


# ---------------------------------------------------------------- inputs
def _grid(case, seed):
    """The padded model: layers of 100 m with seeded resistivities, a resistive block."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x1 = ((np.arange(nx + 1) - nx / 2) * case["hx"]).astype(np.float32)
    x2 = ((np.arange(ny + 1) - ny / 2) * case["hy"]).astype(np.float32)
    x3 = (np.arange(nz + 1) * case["hz"]).astype(np.float32)
    zc = 0.5 * (x3[1:] + x3[:-1]).astype(np.float64)
    floor = 0.0 if case["land"] else 0.15 * nz * case["hz"]
    layer = np.exp(rng.uniform(math.log(1.0 if case["land"] else 0.5), math.log(5.0), size=64))
    rz = np.where(zc < floor, 0.3, layer[np.clip(((zc - floor) / 100.0).astype(int), 0, 63)])
    rho11 = np.empty((nz, ny, nx), np.float32)
    rho33 = np.empty((nz, ny, nx), np.float32)
    rho11[:] = rz.astype(np.float32)[:, None, None]
    rho33[:] = np.where(zc < floor, rz, 1.5 * rz).astype(np.float32)[:, None, None]
    k, j, i = int(nz * rng.uniform(0.3, 0.6)), int(ny * rng.uniform(0.2, 0.5)), int(nx * rng.uniform(0.2, 0.5))
    blk = np.s_[k:k + max(1, nz // 20), j:j + max(1, ny // 4), i:i + max(1, nx // 4)]
    rho11[blk] = rho33[blk] = rng.uniform(20, 100)
    g = cs.Grid.from_arrays(x1, x2, x3, rho11, rho11, rho33).extend(case["nb"], case["lextend"])
    if case["airbc"]:
        g.airbc(case["nfft"], case["nfft"])
    return g, floor


def _freqs(case):
    """Frequencies of the systems: the systems of one frequency next to each other."""
    per = -(-case["nsys"] // case["nfreq"])
    return [FREQS[(5 - s // per) % 6] for s in range(case["nsys"])]


def _vectors(g, case, seed):
    """nsys vectors [Ex | Ey | Ez] on the operator grid, on the GPU."""
    n1, n2, n3 = g.g.n1, g.g.n2, (g.g.nz + g.g.nb if case["airbc"] else g.g.n3)
    dt = torch.complex64 if case["prec"] == 32 else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def fall(n):
        return torch.exp(-5.0 * (torch.arange(n, device="cuda", dtype=torch.float64) / max(1, n - 1) - 0.5).abs())

    parts = []
    for a, b, c in ((n3 + 1, n2 + 1, n1), (n3 + 1, n2, n1 + 1), (n3, n2 + 1, n1 + 1)):
        w = fall(a)[:, None, None] * fall(b)[None, :, None] * fall(c)[None, None, :]
        parts.append(w.reshape(-1))
    w = torch.cat(parts).to(torch.float32 if case["prec"] == 32 else torch.float64)
    x = torch.randn(case["nsys"], w.numel(), dtype=dt, device="cuda", generator=gen)
    return x.mul_(w)


def _pair(case, seed):
    dt = torch.complex64 if case["prec"] == 32 else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["nsys"], case["n"])
    return [torch.randn(shape, dtype=dt, device="cuda", generator=gen) for _ in range(2)]


def _iom(freqs):
    a = np.zeros(2 * len(freqs))
    a[1::2] = [cs.iom_of(f).imag for f in freqs]
    return a


def _dipole(case, floor):
    return np.array([0.25 * case["hx"], 0.25 * case["hy"], max(0.6 * case["hz"], floor - 50.0), 0, 0], np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dot":
        a, b = _pair(case, seed)
        return dict(case=case, a=a, b=b, out=torch.empty(case["nsys"], dtype=torch.complex128, device="cuda"),
                    st=torch.cuda.current_stream().cuda_stream)
    g, floor = _grid(case, seed)
    ctx = cs.Ctx(g, case["airbc"], case["fvm"])
    if kind in ("A", "lusgs", "aphi"):
        x = _vectors(g, case, seed)
        return dict(case=case, ctx=ctx, x=x, y=torch.empty_like(x), iom=_iom(_freqs(case)),
                    st=torch.cuda.Stream())
    if kind == "solve64":
        iom = cs.iom_of(case["freq"])
        return dict(case=case, ctx=ctx, iom=iom, b=ctx.inject_source(iom, ("Ex",), _dipole(case, floor)))
    # sources along x above the seafloor, receivers on it
    half = 0.4 * case["nx"] * case["hx"]
    s0 = _dipole(case, floor)
    per = -(-case["nsys"] // case["nfreq"])
    srcs = np.stack([s0 + np.array([half * (((s % per) + 0.5) / per - 0.5), 0, 0, 0, 0], np.float32)
                     for s in range(case["nsys"])])
    rx = np.linspace(-half, half, 61)
    rec = np.stack([rx, np.zeros(61), np.full(61, max(floor, case["hz"])), np.zeros(61), np.zeros(61)],
                   axis=1).astype(np.float32)
    lo = FREQS.index(case["flow"])
    freqs = [FREQS[min(5, lo + s // per)] for s in range(case["nsys"])]
    return dict(case=case, ctx=ctx, freqs=freqs, srcs=srcs, rec=rec)


# ---------------------------------------------------------------- one pass
def _ptr(t):
    return C.c_void_p(t.data_ptr())


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    L = api.lib()
    if kind == "dot":
        rc = L.csem_cdot_dev(case["prec"], case["n"], case["nsys"], _ptr(s["a"]), _ptr(s["b"]),
                             C.cast(_ptr(s["out"]), C.POINTER(C.c_double)), C.c_void_p(s["st"]))
        if rc:
            raise api.CsemError(rc, L.csem_last_error().decode())
        return s["out"]
    if kind in ("A", "lusgs", "aphi"):
        fn = {"A": L.csem_fdfd_apply_dev, "lusgs": L.csem_lusgs_apply_dev, "aphi": L.csem_aphi_apply_dev}[kind]
        rc = fn(s["ctx"].h, case["prec"], case["nsys"], s["iom"].ctypes.data_as(C.POINTER(C.c_double)), _ptr(s["x"]),
                _ptr(s["y"]), C.c_void_p(s["st"].cuda_stream))
        if rc:
            raise api.CsemError(rc, L.csem_last_error().decode())
        return s["y"]
    if kind == "solve64":
        x, _, _, _ = s["ctx"].solve_fp64(s["iom"], s["b"], algopt=case["algopt"], preco=case["preco"],
                                         niter=case["niter"], tol=1e-8 / case["freq"])
        return x
    r = cs.solve_batch(s["ctx"], s["freqs"], s["srcs"], rec=s["rec"], precision=32, algopt=case["algopt"],
                       niter=case["niter"], max_outer=case["max_outer"],
                       inner_tol=1e-4 if case["max_outer"] == 1 else 0.2)  # a bounded run takes niter iterations
    return r["dcal"].astype(np.complex64)  # as the driver stores and writes them


# ---------------------------------------------------------------- what it cannot do without
def work(case):
    if case["kind"] == "dot":
        bc = 8 if case["prec"] == 32 else 16
        return dict(bytes=2.0 * bc * case["n"] * case["nsys"], flops=8.0 * case["n"] * case["nsys"])
    n1, n2 = case["nx"] + 2 * case["nb"], case["ny"] + 2 * case["nb"]
    n3f = case["nz"] + 2 * case["nb"]
    n3 = case["nz"] + case["nb"] if case["airbc"] else n3f

    def unknowns(k):
        return n1 * (n2 + 1) * (k + 1) + (n1 + 1) * n2 * (k + 1) + (n1 + 1) * (n2 + 1) * k

    N, Nf = unknowns(n3), unknowns(n3f)
    if case["kind"] in ("A", "lusgs", "aphi"):
        bc = 8 if case["prec"] == 32 else 16
        per = {"A": 60.0, "lusgs": 110.0, "aphi": 160.0}[case["kind"]]
        return dict(bytes=2.0 * bc * N * case["nsys"] + bc / 2 * (N if case["kind"] == "A" else Nf),
                    flops=per * N * case["nsys"])
    # Krylov iterations at least: the bounded ones, or 100 of a solve to convergence; each
    # takes two operators and two preconditioners (GMRES: one of each)
    its = min(case["niter"], 100)
    nsys = case.get("nsys", 1)
    bc = 16 if case["kind"] == "solve64" else 8
    ops = 2 if case["algopt"] == 1 else 1
    return dict(bytes=its * nsys * ops * (4.0 * bc * N + bc / 2 * (N + Nf) / nsys), flops=its * nsys * ops * 190.0 * N)


# ---------------------------------------------------------------- the same in 64 bits
class _Geo:
    """The padded model's arrays as tensors."""

    def __init__(self, g, case):
        A, G = g.arrays(), g.g
        self.n1, self.n2, self.n3f, self.nb = G.n1, G.n2, G.n3, G.nb
        self.air, self.fvm = case["airbc"], case["fvm"]
        self.n3 = G.nz + G.nb if self.air else G.n3
        self.ks = G.nb if self.air else 0
        for nm in ("d1", "d2", "d3", "d1s", "d2s", "d3s"):
            setattr(self, nm, torch.from_numpy(A[nm]).cuda())
        n1, n2, n3f = self.n1, self.n2, self.n3f
        self.s1 = torch.from_numpy(A["sigma11"]).cuda().view(n3f + 1, n2 + 1, n1)
        self.s2 = torch.from_numpy(A["sigma22"]).cuda().view(n3f + 1, n2, n1 + 1)
        self.s3 = torch.from_numpy(A["sigma33"]).cuda().view(n3f, n2 + 1, n1 + 1)
        if self.air:
            N1, N2 = G.n1fft, G.n2fft
            self.N1, self.N2 = N1, N2
            self.sH = [torch.from_numpy(A[k]).cuda().view(N2, N1) for k in ("sH1", "sH2")]
            x1, x2, x1s, x2s = A["x1"], A["x2"], A["x1s"], A["x2s"]
            u1, u2 = x1s[0] + np.arange(N1) * G.d1fft, x2s[0] + np.arange(N2) * G.d2fft

            def table(j, w, inside):
                return (torch.from_numpy(np.where(inside, j, 0).astype(np.int64)).cuda(),
                        torch.from_numpy(np.where(inside, w, 0.0)).cuda(), torch.from_numpy(inside * 1.0).cuda())

            self.g1 = table(A["jx"], A["wx"], u1 < x1s[n1 - 1])
            self.g2 = table(A["jy"], A["wy"], u2 < x2s[n2 - 1])

            def back(x, n, d):
                q = (x[:n] - x[0]) / d
                j = q.astype(int)
                return torch.from_numpy(j.astype(np.int64)).cuda(), torch.from_numpy(q - j).cuda()

            self.hx = back(x1, n1 + 1, G.d1fft), back(x2s, n2, G.d2fft)
            self.hy = back(x1s, n1, G.d1fft), back(x2, n2 + 1, G.d2fft)

    def split(self, x, n3):
        n1, n2 = self.n1, self.n2
        a, b = n1 * (n2 + 1) * (n3 + 1), (n1 + 1) * n2 * (n3 + 1)
        return (x[:a].view(n3 + 1, n2 + 1, n1), x[a:a + b].view(n3 + 1, n2, n1 + 1), x[a + b:].view(n3, n2 + 1, n1 + 1))

    def ghosts(self, hz0):
        """Hx, Hy half a cell above the top plane from Hz on it."""
        (j1, w1, m1), (j2, w2, m2) = self.g1, self.g2

        def mix(v, j, w, dim):
            return v.index_select(dim, j) * (1 - w) + v.index_select(dim, j + 1) * w

        K = mix(hz0, j1, w1, 1) * m1
        K = mix(K.t(), j2, w2, 1) * m2
        K = torch.fft.fft2(K.t().contiguous())
        out = []
        for sH, ((p1, q1), (p2, q2)) in ((self.sH[0], self.hx), (self.sH[1], self.hy)):
            U = torch.fft.ifft2(K * sH)
            flat = torch.cat([U.reshape(-1), torch.zeros(self.N1 + 2, dtype=U.dtype, device=U.device)])
            o = 0
            for a, wa in ((0, 1 - q2), (1, q2)):
                for b, wb in ((0, 1 - q1), (1, q1)):
                    o = o + wa[:, None] * wb[None, :] * flat[(p1 + b)[None, :] + self.N1 * (p2 + a)[:, None]]
            out.append(o)
        return out

    def A(self, x, iom):
        n1, n2, n3, ks = self.n1, self.n2, self.n3, self.ks
        Ex, Ey, Ez = self.split(x, n3)
        d1, d1s, d2, d2s = self.d1[:n1], self.d1s[:n1], self.d2[:n2, None], self.d2s[:n2, None]
        d3, d3s = self.d3[ks:ks + n3, None, None], self.d3s[ks:ks + n3, None, None]
        Hx = ((Ez[:, 1:] - Ez[:, :-1]) / d2s - (Ey[1:] - Ey[:-1]) / d3s) / iom
        Hy = ((Ex[1:] - Ex[:-1]) / d3s - (Ez[:, :, 1:] - Ez[:, :, :-1]) / d1s) / iom
        Hz = ((Ey[:, :, 1:] - Ey[:, :, :-1]) / d1s - (Ex[:, 1:] - Ex[:, :-1]) / d2s) / iom
        bx, by, bz = (torch.zeros_like(v) for v in (Ex, Ey, Ez))
        if self.air:
            gx, gy = self.ghosts(Hz[0])
            Hxm, Hym, k0 = torch.cat([gx[None], Hx[:-1]]), torch.cat([gy[None], Hy[:-1]]), 0
        else:
            Hxm, Hym, k0 = torch.cat([Hx[:1], Hx[:-1]]), torch.cat([Hy[:1], Hy[:-1]]), 1
        K = slice(k0, n3)
        D3 = d3[k0:]
        v = (Hz[K, 1:] - Hz[K, :-1]) / d2[1:] - ((Hy[K] - Hym[K]) / D3)[:, 1:n2]
        v = v - self.s1[ks + k0:ks + n3, 1:n2] * Ex[K, 1:n2]
        bx[K, 1:n2] = v * (d1s * d2[1:] * D3 * iom) if self.fvm else v
        v = ((Hx[K] - Hxm[K]) / D3)[:, :, 1:n1] - (Hz[K, :, 1:] - Hz[K, :, :-1]) / d1[1:]
        v = v - self.s2[ks + k0:ks + n3, :, 1:n1] * Ey[K, :, 1:n1]
        by[K, :, 1:n1] = v * (d1[1:] * d2s * D3 * iom) if self.fvm else v
        v = (Hy[:, 1:n2, 1:] - Hy[:, 1:n2, :-1]) / d1[1:] - (Hx[:, 1:, 1:n1] - Hx[:, :-1, 1:n1]) / d2[1:]
        v = v - self.s3[ks:ks + n3, 1:n2, 1:n1] * Ez[:, 1:n2, 1:n1]
        bz[:, 1:n2, 1:n1] = v * (d1[1:] * d2[1:] * d3s * iom) if self.fvm else v
        return torch.cat([v.reshape(-1) for v in (bx, by, bz)])

    def lusgs(self, x, iom):
        """Forward Ex, Ey, Ez, then backward Ez, Ey, Ex: lexicographic Gauss-Seidel sweeps
        from zero, each component coupled to itself in two axes and swept there by
        anti-diagonals; every other term of an update is formed for all points at once."""
        n1, n2, nK = self.n1, self.n2, self.n3f
        up = nK - self.n3
        E = [torch.zeros_like(s, dtype=torch.complex128) for s in (self.s1, self.s2, self.s3)]
        B = [torch.zeros_like(e) for e in E]
        for b, v in zip(B, self.split(x, self.n3)):
            b[up:] = v
        d1, d2, d3 = self.d1[:n1], self.d2[:n2], self.d3[:nK]
        s1, s2, s3 = self.d1s[:n1], self.d2s[:n2], self.d3s[:nK]
        vol1 = s1 * self.d2[:, None][:n2 + 1] * self.d3[:, None, None][:nK + 1]

        def ax(d, s):  # interior points 1..n-1: coupling to the lower and the upper neighbour
            return 1 / (d[1:] * s[:-1]), 1 / (d[1:] * s[1:])

        (l1, u1), (l2, u2), (l3, u3) = ax(d1, s1), ax(d2, s2), ax(d3, s3)
        i1, i2, i3 = slice(1, n1), slice(1, n2), slice(1, nK)
        for comp, fwd in ((0, 1), (1, 1), (2, 1), (2, 0), (1, 0), (0, 0)):
            Ex, Ey, Ez = E
            if comp == 0:
                box, gm, gr, perm = (i3, i2, slice(0, n1)), (l2, u2), (l3, u3), (0, 1, 2)
                sig = self.s1[box]
                dy = (Ey[i3, 1:, 1:] - Ey[i3, 1:, :-1] - Ey[i3, :-1, 1:] + Ey[i3, :-1, :-1]) / d2[1:, None]
                dz = ((Ez[1:, :, 1:] - Ez[1:, :, :-1] - Ez[:-1, :, 1:] + Ez[:-1, :, :-1]) / d3[1:, None, None])[:, i2]
                cross = (dy + dz) / s1
                vol = s1 * d2[1:, None] * d3[1:, None, None]
            elif comp == 1:
                box, gm, gr, perm = (i3, slice(0, n2), i1), (l1, u1), (l3, u3), (0, 2, 1)
                sig = self.s2[box]
                dx = (Ex[i3, 1:, 1:] - Ex[i3, :-1, 1:] - Ex[i3, 1:, :-1] + Ex[i3, :-1, :-1]) / d1[1:]
                dz = (Ez[1:, 1:, i1] - Ez[1:, :-1, i1] - Ez[:-1, 1:, i1] + Ez[:-1, :-1, i1]) / d3[1:, None, None]
                cross = (dx + dz) / s2[:, None]
                vol = (s1[1:] if n1 > 1 else s1) * d2[:, None] * d3[1:, None, None]  # Ex's volume, as the reference
            else:
                box, gm, gr, perm = (slice(0, nK), i2, i1), (l1, u1), (l2, u2), (1, 2, 0)
                sig = self.s3[box]
                dx = (Ex[1:, i2, 1:] - Ex[:-1, i2, 1:] - Ex[1:, i2, :-1] + Ex[:-1, i2, :-1]) / d1[1:]
                dy = (Ey[1:, 1:, i1] - Ey[:-1, 1:, i1] - Ey[1:, :-1, i1] + Ey[:-1, :-1, i1]) / d2[1:, None]
                cross = (dx + dy) / s3[:, None, None]
                vol = s1[1:] * d2[1:, None] * d3[:, None, None]
            own = E[comp]
            rows, march = (gr[0] + gr[1]), (gm[0] + gm[1])
            R, M = rows.numel(), march.numel()
            b, cross, sig, vol = (v.expand(own[box].shape).permute(perm) for v in (B[comp][box], cross, sig, vol))
            f = vol * iom if self.fvm else torch.ones_like(sig)
            aii = (rows[:, None, None] + march[None, :, None]) / iom - sig
            w = 1 / iom / aii
            V = own.permute(perm).contiguous()  # [row][march][line], boundaries included
            rest = b / (f * aii) - w * cross
            if not fwd:
                rest = rest + w * (gm[0][:, None] * V[1:R + 1, 0:M] + gr[0][:, None, None] * V[0:R, 1:M + 1])
            M0 = V.shape[1]
            full = torch.zeros_like(V)
            full[1:R + 1, 1:M + 1] = rest
            W = torch.zeros_like(V)
            W[1:R + 1, 1:M + 1] = w
            P, N = torch.zeros(V.shape[0], M0, 1, dtype=torch.float64, device=V.device), None
            N = torch.zeros_like(P)
            P[:, 1:M + 1] = gm[0 if fwd else 1][None, :, None]
            N[1:R + 1] = gr[0 if fwd else 1][:, None, None]
            Vf, Ff, Wf, Pf, Nf = (t.reshape(V.shape[0] * M0, -1) for t in (V, full, W, P, N))
            step = -1 if fwd else 1
            for t in range(2, R + M + 1) if fwd else range(R + M, 1, -1):
                lo, hi = max(1, t - M), min(R, t - 1)

                def at(z, sh=0):
                    a = t + lo * (M0 - 1) + sh
                    return z[a:a + (hi - lo) * (M0 - 1) + 1:M0 - 1]

                at(Vf)[:] = at(Ff) + at(Wf) * (at(Pf) * at(Vf, step) + at(Nf) * at(Vf, step * M0))
            E[comp] = V.permute([perm.index(a) for a in range(3)]).contiguous()
        return torch.cat([e[up:].reshape(-1) for e in E])


def exact(case, seed):
    kind = case["kind"]
    if kind == "dot":
        a, b = _pair(case, seed)
        return torch.stack([torch.sum(p.to(torch.complex128) * q.to(torch.complex128).conj()) for p, q in zip(a, b)])
    if kind in ("A", "lusgs"):
        g, _ = _grid(case, seed)
        x = _vectors(g, case, seed)
        geo = _Geo(g, case)
        f = geo.A if kind == "A" else geo.lusgs
        return torch.stack([f(v.to(torch.complex128), cs.iom_of(q)) for v, q in zip(x, _freqs(case))])
    if kind == "solve64" and case["niter"] >= 100:  # to convergence, on a model small enough for a dense matrix
        g, floor = _grid(case, seed)
        geo, iom = _Geo(g, case), cs.iom_of(case["freq"])
        ctx = cs.Ctx(g, case["airbc"], case["fvm"])
        b = torch.from_numpy(ctx.inject_source(iom, ("Ex",), _dipole(case, floor))).cuda()
        if b.numel() > 4000:
            return None
        M = torch.stack([geo.A(e, iom) for e in torch.eye(b.numel(), dtype=b.dtype, device="cuda")], 1)
        inner = M.abs().sum(1) > 0  # the boundary rows are zero, and x is zero there
        x = torch.zeros_like(b)
        x[inner] = torch.linalg.solve(M[inner][:, inner], b[inner])
        return x.cpu().numpy()
    return None  # A-phi: sweeps in three axes; the other solves are iterative and most of them bounded
