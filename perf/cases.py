"""The timed cases of the recursive Green-function sweep.

Each case is one call that a user of this package makes: the eigenvalues of one
realization or of a batch of them, the reflection and transmission matrices, the
profiles of the transmission eigenstates, a batch of guides of different sizes,
and the two losses with their gradients with respect to the potential.  Sizes
are those of the repository's own configurations (bench.py, tests): guides of 10
to 512 modes, with the number of slices cut so that a pass stays below a second
(a slice costs the same wherever it lies, so a longer guide repeats the work).
"""
import math
import random

import numpy as np
import torch

import recurgreen_gb300 as rg

# The mode counts of the batched-uneven configuration.
UNEVEN_MODES = (32, 48, 64, 96, 128, 192, 256)


def listed():
    return [
        # the reference's unit of work: one small realization per call, from a seed loop
        dict(name="one_m10", call="one", modes=10, ny=64, nx=200, n=1, dscat=5.0, dabso=0.0, aper=1.0, periodic=False),
        # the small configuration as one batch: 200 realizations of 10 modes
        dict(name="batch_m10", call="tdistrib", modes=10, ny=64, nx=200, n=200, dscat=5.0, dabso=0.0, aper=1.0,
             periodic=False),
        # a ragged medium guide: 37 modes, absorption, part of the aperture, the reference's grid ny = modes
        dict(name="batch_m37_abs", call="tdistrib", modes=37, ny=37, nx=150, n=500, dscat=6.0, dabso=0.4, aper=0.7,
             periodic=False),
        # the width of the reference's own timing remark (wol = 25.5), periodic: t and r of 51 modes for tpattern
        dict(name="rt_m51_periodic", call="rt", modes=51, ny=51, nx=100, n=200, dscat=4.0, dabso=0.0, aper=1.0,
             periodic=True),
        # the batched-uniform configuration: 64 modes, ny = 256
        dict(name="batch_m64", call="tdistrib", modes=64, ny=256, nx=600, n=304, dscat=10.0, dabso=0.0, aper=1.0,
             periodic=False),
        # profiles of the open transmission eigenstates on the same guide
        dict(name="tprofile_m64", call="tprofile", modes=64, ny=256, nx=300, n=152, dscat=10.0, dabso=0.0, aper=1.0,
             periodic=False),
        # t and r of a ragged large guide (tpattern's 'total')
        dict(name="rt_m100_abs", call="rt", modes=100, ny=200, nx=60, n=60, dscat=8.0, dabso=1.0, aper=0.8,
             periodic=False),
        # the differentiation configuration: both losses and both gradients, 128 modes
        dict(name="grads_m128", call="grads", modes=128, ny=512, nx=32, n=64, dscat=5.0, dabso=0.0, aper=1.0,
             periodic=False),
        # the headline guide, one realization per call (the drop-in)
        dict(name="one_m256", call="one", modes=256, ny=1024, nx=60, n=1, dscat=10.0, dabso=0.0, aper=1.0,
             periodic=False),
        # the headline guide, batched
        dict(name="batch_m256", call="tdistrib", modes=256, ny=1024, nx=40, n=152, dscat=10.0, dabso=0.0, aper=1.0,
             periodic=False),
        # the large diffusive configuration: 512 modes, t of a few realizations
        dict(name="t_m512", call="t", modes=512, ny=2048, nx=16, n=16, dscat=20.0, dabso=0.0, aper=1.0,
             periodic=False),
        # the batched-uneven configuration: guides of 32 to 256 modes in one call
        dict(name="uneven", call="multi", modes=0, ny=0, nx=60, n=56, dscat=0.0, dabso=0.0, aper=1.0,
             periodic=False),
    ]


def draw(rng):
    """A case of the same ranges: 5 to 512 modes of any parity, grids of 1 to 4 points per mode, batches of 1 to
    600, absorbing or not, with or without a cut aperture, Dirichlet or (up to 128 modes) periodic."""
    call = rng.choice(["one", "tdistrib", "tdistrib", "tdistrib", "rt", "t", "tprofile", "grads", "multi"])
    if call == "multi":
        return dict(call="multi", modes=0, ny=0, nx=rng.randint(20, 60), n=rng.randint(12, 60), dscat=0.0, dabso=0.0,
                    aper=1.0, periodic=False)
    top = {"one": 256, "tdistrib": 256, "rt": 256, "t": 512, "tprofile": 128, "grads": 160}[call]
    m = int(round(math.exp(rng.uniform(math.log(5), math.log(top)))))
    periodic = call in ("one", "tdistrib", "rt") and m <= 128 and rng.random() < 0.2
    if periodic and m % 2 == 0:
        m += 1
    nx = int(round(math.exp(rng.uniform(math.log(12), math.log(300)))))
    n = 1 if call == "one" else int(round(math.exp(rng.uniform(math.log(4), math.log(600)))))
    if call == "grads":
        n = min(n, 64)

    def seconds():  # a rough upper estimate, to keep a case below the largest listed ones
        slice_s = 1.2e-11 * m ** 3 + 4e-9 * m if m <= 64 else 9e-6 * (m / 128) ** 2.3
        one_s = 3e-6 * m + (2.0e-7 * m ** 1.7 if m <= 64 else 5e-7 * m ** 1.5)
        eig_s = 0.0 if call in ("rt", "t", "grads") else 1.2e-10 * m ** 3
        reps = {"rt": 2.0, "grads": 4.0, "tprofile": 1.3}.get(call, 1.0) * (1.5 if periodic else 1.0)
        return reps * nx * max(n * slice_s, one_s) + max(n * eig_s, 60 * eig_s)

    while seconds() > 0.35:
        if n > 4 and (nx <= 24 or rng.random() < 0.5):
            n = max(4, int(n / 1.5))
        elif nx > 8:
            nx = max(8, int(nx / 1.4))
        else:
            break
    return dict(call=call, modes=m, ny=rng.randint(m, 4 * m), nx=nx, n=n, dscat=round(rng.uniform(1.0, 15.0), 3),
                dabso=0.0 if call == "tprofile" or rng.random() < 0.6 else round(rng.uniform(0.1, 2.0), 3),
                aper=1.0 if call in ("tprofile", "grads") or rng.random() < 0.6 else round(rng.uniform(0.5, 1.0), 3),
                periodic=periodic)


# -- inputs --------------------------------------------------------------------------------------------------------


def _guide(case):
    """Keyword arguments of the guide, with exactly case["modes"] modes."""
    m = case["modes"]
    wol = (m + 0.5) / 2 if not case["periodic"] else (m + 0.5) / 2 - 0.3
    return dict(boundtype="periodic" if case["periodic"] else "dirichlet", nxdiso=case["nx"], nxfree=0, wol=wol,
                exfac=1.0, aratio=1.0, dscat=case["dscat"], dabso=case["dabso"], napera=case["aper"], naperb=1.0,
                ny=case["ny"])


def _seeds(case, seed):
    """Distinct realization seeds; one call's seed lies in the 4096 chunks of its eigenvalue array."""
    r = random.Random(1000003 * seed + 17)
    top = 4096 if case["call"] == "one" else 1 << 24
    return np.array(sorted(r.sample(range(1, top), case["n"])), np.int32)


def _uneven(case, seed):
    """Guides of a batched-uneven call: modes of the configuration's list, up to case["nx"] slices, half of them
    absorbing.  The mix of sizes is the case's; only the realization seeds are the seed's."""
    r = random.Random(7 * case["n"] + case["nx"])
    out = []
    for _ in range(case["n"]):
        m = r.choice(UNEVEN_MODES)
        wol = (m + 0.5) / 2
        out.append(dict(boundtype="dirichlet", nxdiso=r.randint(max(4, case["nx"] // 10), case["nx"]), nxfree=0,
                        wol=wol, exfac=1.0, aratio=1.0, dscat=r.uniform(1, 20),
                        dabso=0.02 * math.pi * wol if r.random() < 0.5 else 0.0, napera=1.0, naperb=1.0, ny=4 * m))
    seeds = random.Random(1000003 * seed + 29).sample(range(1, 1 << 24), case["n"])
    return out, np.array(seeds, np.int32)


def prepare(case, seed):
    if case["call"] == "multi":
        kws, seeds = _uneven(case, seed)
        return dict(case=case, items=[(rg.Waveguide(**kw), int(s)) for kw, s in zip(kws, seeds)])
    w = rg.Waveguide(**_guide(case))
    st = dict(case=case, w=w, seeds=_seeds(case, seed))
    if case["call"] == "one":
        st["tall"] = np.zeros(4096 * w.neigv)
    if case["call"] == "grads":
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
        st["U"] = w.stdu * torch.randn(case["n"], w.nxdiso, w.ny, dtype=torch.float64, device="cuda", generator=g)
    return st


def run(state):
    call = state["case"]["call"]
    if call == "multi":
        return rg.tdistrib_multi(state["items"], return_status=True)
    w, seeds = state["w"], state["seeds"]
    if call == "one":
        s = int(seeds[0])
        w.compute_tdistrib(s, state["tall"])
        return state["tall"][(s - 1) * w.neigv: s * w.neigv]
    if call == "tdistrib":
        return w.tdistrib_batch(seeds)
    if call == "rt":
        return w.refl_trans_v1_batch(seeds)
    if call == "t":
        return w.refl_trans_v1_batch(seeds, want_r=False)[1]
    if call == "tprofile":
        return w.tprofile_batch(seeds, "tprofile", 0.9, 1.0)
    from recurgreen_gb300.adjoint import transmission_losses_and_grads

    return transmission_losses_and_grads(state["U"], w)


# -- work ----------------------------------------------------------------------------------------------------------


def _slice_flops(m, ny, periodic):
    """FP64 operations of one slice: the inverse of a symmetric (4 M^3, or 8 M^3 when periodic) complex matrix, the
    product with the propagator (8 M^3) and the projection of the potential."""
    return (16.0 if periodic else 12.0) * m ** 3 + 2.0 * (2 * m + 1) * ny


def work(case):
    if case["call"] == "multi":
        kws, _ = _uneven(case, 0)
        fl = by = 0.0
        for kw in kws:
            m = int(2 * kw["wol"])
            fl += kw["nxdiso"] * _slice_flops(m, kw["ny"], False)
            by += 4 + 8 * m + 8 * (2 * m + 1) * kw["ny"]
        return {"bytes": by, "flops": fl}
    m, ny, nx, n = case["modes"], case["ny"], case["nx"], case["n"]
    fl = n * nx * _slice_flops(m, ny, case["periodic"])
    by = 4.0 * n + 8.0 * (2 * m + 1) * ny  # seeds and the projection table
    if case["call"] in ("one", "tdistrib"):
        by += 8.0 * n * m
    elif case["call"] in ("rt", "t"):
        by += 16.0 * n * m * m * (2 if case["call"] == "rt" else 1)
        fl += n * nx * 4.0 * m ** 3 if case["call"] == "rt" else 0.0  # r: a second sweep, its inverse only
    elif case["call"] == "tprofile":
        by += 8.0 * n * nx
        fl += 16.0 * n * nx * m * m * 2
    else:  # grads: both columns of G (8 M^3 each) and 16 M^3 per loss and slice; U read, two gradients written
        by += 3 * 8.0 * n * nx * ny
        fl += n * nx * (16.0 + 32.0) * m ** 3
    return {"bytes": by, "flops": fl}


# -- what the calls return, from plain numpy and torch in 64 bits ---------------------------------------------------


class _Guide:
    """The mode set and the slice matrices of a guide (one transverse width, unit length of the disordered part)."""

    def __init__(self, kw):
        wol, nx = kw["wol"], kw["nxdiso"]
        self.per = kw["boundtype"] == "periodic"
        self.kl = 2 * math.pi * wol
        self.nx, self.ny = nx, kw["ny"]
        kdx = self.kl / nx
        if self.per:
            half = int(math.floor(wol))
            ha = int(math.floor(kw["napera"] * wol))
            self.m = 2 * half + 1
            self.rows, self.cols = slice(0, self.m), slice(half - ha, half + ha + 1)
            kp = (np.arange(self.m) - half) / wol
            self.neig = 2 * ha + 1
        else:
            self.m = int(math.floor(2 * wol))
            self.rows, self.cols = slice(0, self.m), slice(0, int(math.floor(2 * kw["napera"] * wol)))
            kp = 0.5 * np.arange(1, self.m + 1) / wol
            self.neig = int(math.floor(2 * kw["napera"] * wol))
        mu = np.sqrt(1 - kp * kp + 1j * kw["dabso"] / self.kl)
        dos = np.sum(np.real(1 / np.sqrt((1 - kp * kp).astype(complex)))) / (wol * (2 * math.pi) ** 2)
        cot = mu / np.tan(mu * kdx)
        self.mu, self.b, self.edge, self.bulk = mu, mu / np.sin(mu * kdx), 1j * mu - cot, -2 * cot
        self.stdu = math.sqrt(kw["dscat"] * self.ny / (2 * math.pi ** 2 * dos * wol * nx))
        y = (np.arange(1, self.ny + 1) - 0.5) / self.ny
        if self.per:
            self.modal = np.exp(2j * math.pi * np.outer(y, kp * wol)) / math.sqrt(self.ny)
        else:
            self.modal = math.sqrt(2 / self.ny) * np.sin(math.pi * np.outer(y, np.arange(1, self.m + 1)))


def _rotl(x, k):
    return (x << np.uint64(k)) | (x >> np.uint64(64 - k))


def _step(s):
    t = s[1] << np.uint64(17)
    s[2] ^= s[0]
    s[3] ^= s[1]
    s[1] ^= s[2]
    s[0] ^= s[3]
    s[2] ^= t
    s[3] = _rotl(s[3], 45)


def _next(s):
    out = _rotl(s[1] * np.uint64(5), 7) * np.uint64(9)
    _step(s)
    return out


def _bits(s):
    """(4, n) words as an (n, 256) matrix of 0 and 1."""
    return ((s.T[:, :, None] >> np.arange(64, dtype=np.uint64)) & np.uint64(1)).reshape(s.shape[1], 256).astype(np.float32)


def _words(b):
    v = b.reshape(-1, 4, 64).astype(np.uint64) << np.arange(64, dtype=np.uint64)
    return np.ascontiguousarray(v.sum(axis=2, dtype=np.uint64).T)


def _potentials(g, seeds):
    """The potentials of the seeds, (n, nx, ny): normals by Box-Muller from xoshiro256** seeded by eight numbers of an
    ANSI-C generator; along x first, so column iy starts 2 nx iy draws into a seed's stream."""
    with np.errstate(over="ignore"):
        s, put = np.asarray(seeds).astype(np.uint32), []
        for _ in range(8):
            s = s * np.uint32(1103515245) + np.uint32(12345)
            put.append(s.astype(np.uint64))
        keys = (0xbd0c5b6e50c2df49, 0xd46061cd46e1df38, 0xbb4f4d4ed6103544, 0x114a583d0756ad39)
        start = np.stack([(put[7 - 2 * k] | (put[6 - 2 * k] << np.uint64(32))) ^ np.uint64(keys[k]) for k in range(4)])
        unit = _words(np.eye(256, dtype=np.float32))  # the generator is linear over GF(2)
        for _ in range(2 * g.nx):
            _step(unit)
        jump = _bits(unit)
        cols, b = [], _bits(start)
        for _ in range(g.ny):
            cols.append(_words(b))
            b = np.mod(b @ jump, 2)
        st = np.stack(cols, axis=2)  # (4, n, ny)
        out = np.empty((len(seeds), g.nx, g.ny))
        for ix in range(g.nx):
            u1 = (_next(st) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
            u2 = (_next(st) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
            out[:, ix] = g.stdu * np.sqrt(-2 * np.log(u1)) * np.cos(2 * math.pi * u2)
    return out


def _sweep(g, U, reverse=False, states=None):
    """(Gss, Gs1) after the last slice for the potentials U (n, nx, ny), torch complex128."""
    dev = U.device
    b = torch.from_numpy(g.b).to(dev)
    modal = torch.from_numpy(g.modal).to(dev)
    eye = torch.eye(g.m, dtype=torch.complex128, device=dev)
    gss = gs1 = None
    for k in range(g.nx):
        n = g.nx - 1 - k if reverse else k
        v = (modal.conj().T * U[:, n, None, :]) @ modal
        x = torch.diag(torch.from_numpy(g.edge if k in (0, g.nx - 1) else g.bulk).to(dev)) - v
        if gss is None:
            gss = torch.linalg.inv(x)
            gs1 = gss @ eye
        else:
            gss = torch.linalg.inv(x - b[:, None] * gss * b)
            gs1 = -gss @ (b[:, None] * gs1)
        if states is not None:
            states.append((gss, gs1))
    return gss, gs1


def _tmat(g, gs1, real):
    mu = np.sqrt(np.real(g.mu)).astype(complex) if real else np.sqrt(g.mu)
    s = torch.from_numpy(mu).to(gs1.device)
    return 2j * s[:, None] * gs1 * s


def _eigs(g, t):
    return torch.linalg.svdvals(t.cpu())[..., : g.neig] ** 2


def _too_long(case):
    """The plain version takes over about 20 seconds: many slices of large matrices, on cuSOLVER."""
    return case["n"] * case["nx"] * (case["modes"] / 64.0) ** 2 > 4e5


def exact(case, seed):
    if case["call"] == "multi":
        kws, seeds = _uneven(case, seed)
        out = []
        for kw, s in zip(kws, seeds):
            g = _Guide(kw)
            U = torch.from_numpy(_potentials(g, [s])).cuda()
            out.append(_eigs(g, _tmat(g, _sweep(g, U)[1], False))[0].numpy())
        return out, None
    if _too_long(case):
        return None
    g = _Guide(_guide(case))
    if case["call"] == "grads":
        U = prepare(case, seed)["U"].clone().requires_grad_(True)
        t = _tmat(g, _sweep(g, U)[1], False)[:, g.rows, g.cols]
        l1 = (t.abs() ** 2).sum((1, 2))
        l2 = ((t.conj().transpose(1, 2) @ t).abs() ** 2).sum((1, 2))
        d1, = torch.autograd.grad(l1.sum(), U, retain_graph=True)
        d2, = torch.autograd.grad(l2.sum(), U)
        return l1.detach(), l2.detach(), d1, d2
    U = torch.from_numpy(_potentials(g, _seeds(case, seed))).cuda()
    if case["call"] in ("rt", "t"):
        t = _tmat(g, _sweep(g, U)[1], True).cpu().numpy()
        if case["call"] == "t":
            return t
        r = _tmat(g, _sweep(g, U, reverse=True)[0], True).cpu().numpy() - np.eye(g.m)
        return r, t
    if case["call"] == "tprofile":
        states = []
        t = _tmat(g, _sweep(g, U, states=states)[1], True)
        _, sv, vh = torch.linalg.svd(t.cpu())  # on the CPU: cuSOLVER's batched eigenvectors stop at 1e-8
        T, V = (sv ** 2).cuda(), vh.conj().transpose(1, 2).cuda()
        keep = (T >= 0.9) & (T <= 1.0)
        nt = keep.sum(1)
        w = torch.from_numpy(np.sqrt(np.real(g.mu)).astype(complex)).cuda()[:, None] * V * keep[:, None, :]
        b = torch.from_numpy(g.b).cuda()[:, None]
        prof = torch.zeros(case["n"], g.nx, dtype=torch.float64, device="cuda")
        y = None
        for n in reversed(range(g.nx)):
            s, z = states[n]
            y = z @ w if y is None else z @ w - s @ (b * y)
            prof[:, n] = (y.abs() ** 2).sum((1, 2))
        prof *= (4.0 / nt.clamp(min=1).double())[:, None]
        return prof[:, None, :].cpu().numpy(), nt[:, None].to(torch.int32).cpu().numpy(), T.mean(1).cpu().numpy()
    t = _tmat(g, _sweep(g, U)[1], False)[:, g.rows, g.cols]
    return _eigs(g, t).reshape(-1).numpy()
