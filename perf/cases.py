"""What the framework is used for, as cases that can be timed and checked.

Every case is a call (or the short chain of calls) a user's program makes:
  block     GpuBlock: a state that lies on the device goes in
            (upload_device, set_time), some cycles run, the state comes back
            into device arrays with its time and next time step
  ensemble  Ensemble: some more cycles of every box, then every box's state
  learned   a GpuBlock of the learned order, as a block case
  grad      Trainer.grad: loss and gradients of one batch
  train     Trainer: weights set, some training steps, weights, losses and
            feature range back

The initial states are the workloads' (Orszag-Tang-like vortices, the MHD
rotor, decaying turbulence, the low-beta box), seeded.  `exact` restates the
scheme (and the network) in plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import idefix_gb300 as ig
from idefix_gb300 import learned

DEVICE = "cuda"
F64 = torch.float64
GAMMA = 5.0 / 3.0
NIN, NH, NOUT = 216, 128, 16
RANGE = 2.5  # trained feature range handed to the learned order


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _block(name, dims, nx, ny, nz, ic, cycles, precision="fp64", order="plm", solver="hlld", emf="uct_contact",
           nstages=2, cfl=0.6, walls="periodic", autotune=False, kind="block"):
    return {"name": name, "kind": kind, "dims": dims, "nx": nx, "ny": ny, "nz": nz, "ic": ic, "cycles": cycles,
            "precision": precision, "order": order, "solver": solver, "emf": emf, "nstages": nstages, "cfl": cfl,
            "walls": walls, "autotune": autotune}


def listed():
    return [
        # one TimeIntegrator::Cycle of the smallest ensemble box as a block: launches and latency
        _block("ot2d_64_fp64_cycle", 2, 64, 64, 1, "vortex", 1),
        # the 2-D Orszag-Tang problem at the reference's size, a stretch of its run to t = 0.5
        _block("ot2d_256_fp64", 2, 256, 256, 1, "vortex", 8),
        # the MHD rotor at the reference's settings (outflow walls, Roe), the mixed path in 2-D
        _block("rotor2d_512_roe_mixed", 2, 512, 512, 1, "rotor", 4, precision="mixed", solver="roe", cfl=0.2,
               walls="outflow"),
        # a coarse 3-D run (the learned workload's plain run at twice its resolution)
        _block("turb3d_64_fp64", 3, 64, 64, 64, "turbulence", 2),
        # the headline workload: 3-D decaying turbulence 256^3, one RK2 cycle
        _block("turb3d_256_fp64", 3, 256, 256, 256, "turbulence", 1, autotune=True),
        # the same workload on the mixed path
        _block("turb3d_256_mixed", 3, 256, 256, 256, "turbulence", 4, precision="mixed", autotune=True),
        # the low-beta precision workload (LimO3) on the mixed path, at half its edge length
        _block("lowbeta3d_192_limo3_mixed", 3, 192, 192, 192, "lowbeta", 4, precision="mixed", order="limo3",
               autotune=True),
        # a box of odd sizes, another scheme of the test matrix (PPM, HLL, arithmetic EMFs, RK3)
        _block("box3d_odd_ppm_hll_fp64", 3, 91, 62, 45, "turbulence", 1, order="ppm", solver="hll",
               emf="arithmetic", nstages=3, cfl=0.4),
        # the learned interface-state correction at its coarse size
        _block("learned3d_32_fp64", 3, 32, 32, 32, "turbulence", 2, order="learned", kind="learned"),
        # a share of the 512-box ensemble of uneven 2-D boxes
        {"name": "ensemble2d_48_fp64", "kind": "ensemble", "boxes": 48, "cycles": 2, "precision": "fp64",
         "smallest": 64, "largest": 512},
        # one batch's gradients, as a training loop outside the library asks for them
        {"name": "mlp_grad_8192", "kind": "grad", "batch": 8192},
        # the training loop of the correction network
        {"name": "mlp_train_8192", "kind": "train", "batch": 8192, "steps": 16, "snapshots": 8, "nc": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """one more case: mostly single blocks, in the proportion the listed ones have"""
    kind = rng.choice(["2d", "2d", "3d", "3d", "3d", "learned", "ensemble", "grad", "train"])
    if kind == "grad":
        return {"kind": "grad", "batch": _log_int(rng, 256, 8192)}
    if kind == "train":
        return {"kind": "train", "batch": _log_int(rng, 256, 8192), "steps": rng.randint(2, 16),
                "snapshots": rng.randint(2, 8), "nc": rng.choice([12, 16, 27, 32])}
    if kind == "ensemble":
        return {"kind": "ensemble", "boxes": _log_int(rng, 2, 40), "cycles": rng.randint(1, 3),
                "precision": rng.choice(["fp64", "mixed"]), "smallest": rng.choice([64, 96]),
                "largest": rng.choice([128, 256, 384])}
    if kind == "learned":
        n = [_log_int(rng, 12, 40) for _ in range(3)]
        c = _block("", 3, n[0], n[1], n[2], "turbulence", rng.randint(1, 2), order="learned", kind="learned")
    else:
        prec = rng.choice(["fp64", "mixed"])
        order = rng.choice(["plm", "plm", "limo3", "ppm"])
        solver = rng.choice(["hlld", "hlld", "roe", "hll"])
        emf = rng.choice(["uct_contact", "uct_contact", "arithmetic"])
        nst = rng.choice([2, 2, 3])
        if kind == "2d":
            n = [_log_int(rng, 48, 520) for _ in range(2)]
            ic = rng.choice(["vortex", "vortex", "rotor"])
            c = _block("", 2, n[0], n[1], 1, ic, rng.randint(1, 8), precision=prec, order=order, solver=solver,
                       emf=emf, nstages=nst, cfl=0.2 if ic == "rotor" else 0.4,
                       walls="outflow" if ic == "rotor" else "periodic")
        else:
            n = [_log_int(rng, 16, 200 if prec == "mixed" else 110) for _ in range(3)]
            c = _block("", 3, n[0], n[1], n[2], rng.choice(["turbulence", "turbulence", "lowbeta"]),
                       rng.randint(1, 2), precision=prec, order=order, solver=solver, emf=emf, nstages=nst, cfl=0.4,
                       autotune=rng.random() < 0.4)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# initial states (device, reference layout)
# ---------------------------------------------------------------------------
def _ng(case):
    return 3 if case["order"] == "ppm" else 2


def _domain(case):
    """cell widths: the unit box along x, square cells (the rotor's box is [-0.5, 0.5]^2)"""
    return [1.0 / case["nx"]] * 3


def _extent(case):
    dx = _domain(case)
    n = (case["nx"], case["ny"], case["nz"])
    return tuple(dx[d] * n[d] for d in range(3))


def _smooth(gen, shape, kmax):
    """Gaussian field on a periodic grid, power ~ k^-2 on 1 <= |k| <= kmax, unit rms; shape (k, j, i)"""
    m = [max(1, min(kmax, n // 4)) if n > 1 else 0 for n in shape]
    spec = torch.zeros((shape[0], shape[1], shape[2] // 2 + 1), dtype=torch.complex128)
    low = torch.randn((2 * kmax + 1, 2 * kmax + 1, kmax + 1, 2), generator=gen, dtype=F64)
    ks = [torch.arange(-m[0], m[0] + 1), torch.arange(-m[1], m[1] + 1), torch.arange(0, m[2] + 1)]
    k2 = (ks[0][:, None, None] ** 2 + ks[1][None, :, None] ** 2 + ks[2][None, None, :] ** 2).to(F64)
    amp = torch.where(k2 > 0, k2.clamp(min=1.0) ** -1.0, torch.zeros_like(k2)) * (k2 <= kmax * kmax)
    part = torch.view_as_complex(low)[kmax - m[0]:kmax + m[0] + 1, kmax - m[1]:kmax + m[1] + 1, :m[2] + 1] * amp
    spec[(ks[0] % shape[0])[:, None, None], (ks[1] % shape[1])[None, :, None], ks[2][None, None, :]] = part
    a = torch.fft.irfftn(spec.to(DEVICE), s=shape, dim=(0, 1, 2))
    return a / a.square().mean().sqrt()


def _wrapped(n, ng, extra=0):
    return (torch.arange(n + 2 * ng + extra, device=DEVICE) - ng) % n


def _cells(case, fields):
    """active-cell fields (k, j, i) -> ghosted [len(fields), nt2, nt1, nt0], periodic ghosts"""
    g, D = _ng(case), case["dims"]
    n = (case["nx"], case["ny"], case["nz"])
    ix = [_wrapped(n[d], g) if d < D else torch.zeros(1, dtype=torch.long, device=DEVICE) for d in range(3)]
    a = torch.stack([f.expand(n[2], n[1], n[0]) for f in fields])
    return a[:, ix[2][:, None, None], ix[1][None, :, None], ix[0][None, None, :]].contiguous()


def _faces(case, fields):
    """periodic left-face fields -> ghosted Vs"""
    g, D = _ng(case), case["dims"]
    n = (case["nx"], case["ny"], case["nz"])
    ix = [_wrapped(n[d], g, 1) if d < D else torch.zeros(1, dtype=torch.long, device=DEVICE) for d in range(3)]
    a = torch.stack([f.expand(n[2], n[1], n[0]) for f in fields])
    return a[:, ix[2][:, None, None], ix[1][None, :, None], ix[0][None, None, :]].contiguous()


def _axis(n, d):
    x = (torch.arange(n, dtype=F64, device=DEVICE) + 0.5) / n
    return x.view([-1 if 2 - d == a else 1 for a in range(3)])


def _initial(case, seed):
    gen = torch.Generator().manual_seed(int(seed))
    D = case["dims"]
    n = (case["nx"], case["ny"], case["nz"])
    shape = (n[2], n[1], n[0])
    dx = _domain(case)
    one = torch.ones(shape, dtype=F64, device=DEVICE)
    if case["ic"] == "vortex":  # Orszag-Tang-like: Mach U[0.5, 2], beta log-U[0.1, 10], shifted phases
        u = torch.rand(4, generator=gen, dtype=F64).tolist()
        return _vortex(case, 0.5 + 1.5 * u[0], 10.0 ** (2.0 * u[1] - 1.0), u[2], u[3])
    if case["ic"] == "rotor":  # the disc a little off the centre, as a seeded family of the test problem
        u = (torch.rand(3, generator=gen, dtype=F64) - 0.5).tolist()
        x = (_axis(n[0], 0) - 0.5 - 0.1 * u[0]) * (dx[0] * n[0])
        y = (_axis(n[1], 1) - 0.5 - 0.1 * u[1]) * (dx[1] * n[1])
        r = (x * x + y * y).sqrt()
        f = ((0.115 - r) / 0.015).clamp(0.0, 1.0)
        om = 20.0 * (1.0 + 0.2 * u[2])
        vphi = om * torch.where(r < 0.1, r, f * 0.1)
        V = [1.0 + 9.0 * f, -y / r * vphi, x / r * vphi, one]
        B = [one * (5.0 / math.sqrt(4.0 * math.pi)), 0.0 * one]
        Vc = torch.cat([_cells(case, V), torch.zeros((2,) + _cells(case, V[:1]).shape[1:], dtype=F64, device=DEVICE)])
        return Vc.contiguous(), _faces(case, B)
    if case["ic"] == "turbulence":
        v = [_smooth(gen, shape, 8) for _ in range(3)]
        s = 1.0 / math.sqrt(float(sum(c.square().mean() for c in v)))
        A = [_smooth(gen, shape, 8) for _ in range(3)]
        roll = lambda a, d: torch.roll(a, -1, dims=2 - d)  # noqa: E731
        dif = lambda a, d: (roll(a, d) - a) / dx[d]        # noqa: E731
        B = [dif(A[2], 1) - dif(A[1], 2), dif(A[0], 2) - dif(A[2], 0), dif(A[1], 0) - dif(A[0], 1)]
        p0, b0, beta = 1.0 / GAMMA, 0.1, 10.0
        sb = math.sqrt((2.0 * p0 / beta - b0 * b0) / float(sum(c.square().mean() for c in B)))
        B = [B[0] * sb + b0, B[1] * sb, B[2] * sb]
        V = [one] + [c * s for c in v] + [one * p0]
    else:  # low beta: uniform Bz = 1, p = beta B^2 / 2
        beta, mach = 1e-3, 0.3
        rho = 1.0 + 0.1 * _smooth(gen, shape, 4)
        v = [_smooth(gen, shape, 4) for _ in range(3)]
        s = mach * math.sqrt(GAMMA * 0.5 * beta) / math.sqrt(float(sum(c.square().mean() for c in v)))
        V = [rho] + [c * s for c in v] + [one * (0.5 * beta)]
        B = [0.0 * one, 0.0 * one, one]
    Vc = torch.cat([_cells(case, V), torch.zeros_like(_cells(case, V[:D]))])
    return Vc.contiguous(), _faces(case, B)


def _vortex(case, mach, beta, px, py):
    n = (case["nx"], case["ny"], 1)
    one = torch.ones((1, n[1], n[0]), dtype=F64, device=DEVICE)
    x, y = _axis(n[0], 0) + px, _axis(n[1], 1) + py
    p, rho = 5.0 / (12.0 * math.pi), 25.0 / (36.0 * math.pi)
    cs, B0 = math.sqrt(GAMMA * p / rho), math.sqrt(2.0 * p / beta)
    V = [rho * one, -mach * cs * torch.sin(2 * math.pi * y) * one, mach * cs * torch.sin(2 * math.pi * x) * one, p * one]
    B = [-B0 * torch.sin(2 * math.pi * y) * one, B0 * torch.sin(4 * math.pi * x) * one]
    Vc = torch.cat([_cells(case, V), torch.zeros_like(_cells(case, V[:2]))])
    return Vc.contiguous(), _faces(case, B)


def _dt0(case):
    return 0.03 / case["nx"]


def _params(seed):
    """a network as a training run leaves it: He-scaled layers, a small output layer"""
    rng = np.random.default_rng(seed)
    p = learned.init_params(seed=int(rng.integers(1 << 30)), out_scale=0.02)
    for o, m in ((NIN * NH, NH), (NIN * NH + NH + NH * NH, NH)):
        p[o:o + m] = 0.05 * rng.standard_normal(m)
    return p.astype(np.float32)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _kwargs(case):
    D = case["dims"]
    n = (case["nx"], case["ny"], case["nz"])[:D]
    kw = dict(dims=D, n=n, xend=_extent(case), order=case["order"], solver=case["solver"], emf=case["emf"],
              nstages=case["nstages"], cfl=case["cfl"], first_dt=_dt0(case), precision=case["precision"])
    if case["walls"] == "outflow":
        kw["bc"] = (("outflow", "outflow"),) * D
    return kw


def _ensemble_boxes(case, seed):
    """(block case, mach, beta) per box: sizes of the ensemble workload within the case's bounds"""
    rng = np.random.default_rng(seed)
    sizes = [s for s in (64, 96, 128, 192, 256, 384, 512) if case["smallest"] <= s <= case["largest"]]
    boxes = []
    for b in range(case["boxes"]):  # every seed has the same sizes, in another order
        n = sizes[b % len(sizes)]
        boxes.append(_block("", 2, n, n, 1, "vortex", case["cycles"], precision=case["precision"]))
    order = rng.permutation(len(boxes))
    mach, beta = rng.uniform(0.5, 2.0, len(boxes)), 10.0 ** rng.uniform(-1.0, 1.0, len(boxes))
    return [(boxes[o], float(mach[k]), float(beta[k])) for k, o in enumerate(order)]


def _batch(case, seed):
    """features near what a stencil of a smooth state gives, targets of the corrections' size"""
    g = torch.Generator().manual_seed(int(seed))
    B = case["batch"]
    X = torch.zeros((B, learned.K1), dtype=torch.float32)
    X[:, :NIN] = 0.3 * torch.randn((B, NIN), generator=g)
    T = 0.05 * torch.randn((B, NOUT), generator=g) + 0.1 * X[:, :NOUT]
    return X.to(DEVICE).to(torch.bfloat16).contiguous(), T.to(DEVICE).contiguous()


def _dataset(case, seed):
    """coarse snapshots (float32 primitives) and their face targets"""
    g = torch.Generator().manual_seed(int(seed))
    S, nc = case["snapshots"], case["nc"]
    P = torch.empty((S, 8, nc, nc, nc), dtype=torch.float32, device=DEVICE)
    for s in range(S):
        f = [_smooth(g, (nc, nc, nc), 4) for _ in range(8)]
        for v, (mean, amp) in enumerate(((1.0, 0.1), (0, 0.5), (0, 0.5), (0, 0.5), (0.6, 0.06), (0.1, 0.2), (0, 0.2),
                                         (0, 0.2))):
            P[s, v] = (mean + amp * f[v]).float()
        P[s, 0].clamp_(min=0.3)
        P[s, 4].clamp_(min=0.2)
    T = torch.empty((S, 3, 16, nc ** 3), dtype=torch.float32, device=DEVICE)
    for d in range(3):
        for r in range(8):
            q = P[:, _rot(r, d)]
            a, b = torch.roll(q, 1, 3 - d), torch.roll(q, -1, 3 - d)
            T[:, d, r] = (0.5 * (a + q) - 0.0625 * (b - q)).reshape(S, -1)
            T[:, d, 8 + r] = (0.5 * (q + b) - 0.0625 * (a - q)).reshape(S, -1)
    return P, T


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return {"case": case, "trainer": learned.Trainer(max_batch=case["batch"], params=_params(seed)),
                "batch": _batch(case, seed)}
    if kind == "train":
        P, T = _dataset(case, seed)
        torch.cuda.synchronize()
        tr = learned.Trainer(max_batch=case["batch"], params=_params(seed))
        tr.set_dataset(P, T)
        return {"case": case, "trainer": tr, "params": _params(seed), "seed": int(seed)}
    if kind == "ensemble":
        boxes = _ensemble_boxes(case, seed)
        ens = ig.Ensemble([_kwargs(c) for c, _, _ in boxes])
        out = []
        for b, (c, mach, beta) in enumerate(boxes):
            Vc, Vs = _vortex(c, mach, beta, 0.0, 0.0)
            ens.upload(b, Vc.cpu().numpy(), Vs.cpu().numpy())
            out.append((torch.empty_like(Vc), torch.empty_like(Vs)))
        return {"case": case, "ensemble": ens, "out": out}
    Vc, Vs = _initial(case, seed)
    blk = ig.GpuBlock(**_kwargs(case))
    if kind == "learned":
        blk.set_learned(_params(seed), -RANGE * np.ones(NIN, np.float32), RANGE * np.ones(NIN, np.float32))
    torch.cuda.synchronize()
    if case["autotune"]:  # as the workloads do for a long run: the state only has to be a real one
        blk.upload_device(Vc.data_ptr(), Vs.data_ptr())
        blk.autotune(1)
    return {"case": case, "block": blk, "in": (Vc, Vs), "out": (torch.empty_like(Vc), torch.empty_like(Vs))}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "grad":
        g, loss = state["trainer"].grad(*state["batch"])
        return {"grad": g, "loss": np.float64(loss)}
    if kind == "train":
        tr = state["trainer"]
        tr.set_params(state["params"])
        losses = tr.train(case["steps"], case["batch"], lr=2e-3, lr_end=2e-5, seed=state["seed"])
        lo, hi = tr.feature_range()
        return {"params": tr.get_params(), "losses": losses, "lo": lo, "hi": hi}
    if kind == "ensemble":
        ens = state["ensemble"]
        ens.run(max_cycles=case["cycles"])
        for b, (Vc, Vs) in enumerate(state["out"]):
            ens.download_device(b, Vc.data_ptr(), Vs.data_ptr())
        return {"Vc": torch.cat([v.view(-1) for v, _ in state["out"]]),
                "Vs": torch.cat([v.view(-1) for _, v in state["out"]])}
    blk = state["block"]
    blk.upload_device(state["in"][0].data_ptr(), state["in"][1].data_ptr())
    blk.set_time(0.0, _dt0(case), 0)
    blk.run(max_cycles=case["cycles"])
    blk.download_device(state["out"][0].data_ptr(), state["out"][1].data_ptr())
    t, dt, _ = blk.get_time()
    return {"Vc": state["out"][0], "Vs": state["out"][1], "time": np.array([t, dt])}


def work(case):
    """bytes: every input and output once; flops: the scheme's operations per zone, cycle and stage
    (counted per zone-cycle of RK2: 3380 in 3-D and 1740 in 2-D with PLM and HLLD), the network's products"""
    kind = case["kind"]
    mac = NIN * NH + NH * NH + NH * NOUT
    if kind == "grad":
        B = case["batch"]
        return {"bytes": B * (learned.K1 * 2 + NOUT * 4) + 2 * learned.NPARAM * 4, "flops": 6.0 * mac * B}
    if kind == "train":
        B = case["batch"] * case["steps"]
        return {"bytes": B * (NIN + NOUT) * 4 + 2 * learned.NPARAM * 4, "flops": 6.0 * mac * B}
    if kind == "ensemble":
        boxes = [c for c, _, _ in _ensemble_boxes(case, 0)]
        cells = sum(c["nx"] * c["ny"] for c in boxes)
        return {"bytes": 2.0 * cells * 8 * 8, "flops": 1740.0 * cells * case["cycles"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    D = case["dims"]
    fl = (3380.0 if D == 3 else 1740.0) * case["nstages"] / 2 * cells * case["cycles"]
    if kind == "learned":
        fl += 2.0 * mac * 3 * case["nstages"] * cells * case["cycles"]
    return {"bytes": 2.0 * cells * (3 * D + 2) * 8, "flops": fl}


# ---------------------------------------------------------------------------
# the scheme in plain torch, 64 bits.  Arrays are [.., k, j, i]; direction d is
# axis -1 - d.
# ---------------------------------------------------------------------------
def _sl(a, d, lo, hi):
    return a.narrow(a.dim() - 1 - d, lo, hi - lo)


def _minmod0(a, b):
    return torch.where(a * b > 0, 2 * a * b / torch.where(a + b != 0, a + b, torch.ones_like(a)), torch.zeros_like(a))


def _limo3(dp, dm, dx):
    th = dm / (dp + 1e-16)
    q = (2 + th) / 3
    z = torch.zeros_like(q)
    psi = torch.maximum(z, torch.minimum(q, torch.maximum(-0.5 * th, torch.minimum(
        q, torch.minimum(torch.full_like(q, 1.5), 2 * th)))))
    eta = (dm * dm + dp * dp) / (0.1 * dx) ** 2
    e = 1e-12
    mid = 0.5 * ((1 - (eta - 1) / e) * q + (1 + (eta - 1) / e) * psi)
    return torch.where(eta <= 1 - e, q, torch.where(eta >= 1 + e, psi, mid))


def _ppm_face(vm1, v0, vp1, vp2, f):
    dl, dc, dr = vm1 - 2 * v0 + vp1, 3 * (v0 - 2 * f + vp1), v0 - 2 * vp1 + vp2
    same = (dl.sign() == dc.sign()) & (dr.sign() == dc.sign())
    d = torch.where(same, dc.sign() * torch.minimum(1.25 * torch.minimum(dl.abs(), dr.abs()), dc.abs()),
                    torch.zeros_like(dc))
    return torch.where((vp1 - f) * (f - v0) < 0, 0.5 * (v0 + vp1) - d / 6, f)


def _ppm(w):
    vm2, vm1, v0, vp1, vp2 = w
    vr = 7 / 12 * (v0 + vp1) - 1 / 12 * (vm1 + vp2)
    vl = 7 / 12 * (vm1 + v0) - 1 / 12 * (vm2 + vp1)
    vl = _ppm_face(vm2, vm1, v0, vp1, vl)
    vr = _ppm_face(vm1, v0, vp1, vp2, vr)
    f = 6 * (vl + vr - 2 * v0)
    c0, cp, cm = vm1 + vp1 - 2 * v0, v0 + vp2 - 2 * vp1, vm2 + v0 - 2 * vm1
    same = (f.sign() == c0.sign()) & (f.sign() == cp.sign()) & (f.sign() == cm.sign())
    q = torch.where(same, f.sign() * torch.minimum(f.abs(), 1.25 * torch.minimum(
        cm.abs(), torch.minimum(c0.abs(), cp.abs()))), torch.zeros_like(f))
    big = torch.maximum(torch.maximum(vm1.abs(), v0.abs()), vp1.abs())
    rho = torch.where(f.abs() > 1e-12 * big, q / torch.where(f != 0, f, torch.ones_like(f)), torch.zeros_like(f))
    ext = ((vr - v0) * (v0 - vl) <= 0) | ((vm1 - v0) * (v0 - vp1) <= 0)
    lim = rho <= 1 - 1e-12
    l1, r1 = torch.where(lim, v0 - rho * (v0 - vl), vl), torch.where(lim, v0 + rho * (vr - v0), vr)
    r2 = torch.where((vr - v0).abs() >= 2 * (v0 - vl).abs(), v0 + 2 * (v0 - vl), vr)
    l2 = torch.where((vl - v0).abs() >= 2 * (v0 - r2).abs(), v0 + 2 * (v0 - r2), vl)
    return torch.where(ext, l1, l2), torch.where(ext, r1, r2)


def _recon(order, V, d, beg, end, dx, positive):
    """left-face and right-face states of the cells beg - 1 .. end along d"""
    at = lambda o: _sl(V, d, beg - 1 + o, end + 1 + o)  # noqa: E731
    w1, dm, dp = at(0), at(0) - at(-1), at(1) - at(0)
    if order == "ppm":
        vl, vr = _ppm([at(o) for o in (-2, -1, 0, 1, 2)])
        if positive:
            h = 0.5 * _minmod0(dp, dm)
            vl, vr = torch.where(vl <= 0, w1 - h, vl), torch.where(vr <= 0, w1 + h, vr)
        return vl, vr
    if order == "limo3":
        vr = w1 + 0.5 * dp * _limo3(dp, dm, dx)
        vl = w1 - 0.5 * dm * _limo3(dm, dp, dx)
        if positive:  # the minmod slope of the positivity fallback is zero
            vl, vr = torch.where(vl <= 0, w1, vl), torch.where(vr <= 0, w1, vr)
        return vl, vr
    h = 0.5 * _minmod0(dp, dm)
    return w1 - h, w1 + h


def _cons(V, D):
    kin = sum(V[1 + c] ** 2 for c in range(D))
    mag = sum(V[D + 2 + c] ** 2 for c in range(D))
    E = V[D + 1] / (GAMMA - 1) + 0.5 * V[0] * kin + 0.5 * mag
    return [V[0]] + [V[0] * V[1 + c] for c in range(D)] + [E] + [V[D + 2 + c] for c in range(D)]


def _flux(V, U, D, d):
    vn, bn = V[1 + d], V[D + 2 + d]
    pt = V[D + 1] + 0.5 * sum(V[D + 2 + c] ** 2 for c in range(D))
    vB = sum(V[1 + c] * V[D + 2 + c] for c in range(D))
    F = [U[1 + d]] + [U[1 + c] * vn - bn * V[D + 2 + c] + (pt if c == d else 0.0) for c in range(D)]
    F += [(U[D + 1] + pt) * vn - bn * vB]
    return F + [vn * V[D + 2 + c] - bn * V[1 + c] if c != d else torch.zeros_like(vn) for c in range(D)]


def _fast(V, D, d):
    gp = GAMMA * V[D + 1]
    bt = sum(V[D + 2 + c] ** 2 for c in range(D) if c != d)
    b = bt + V[D + 2 + d] ** 2
    return ((gp + b + ((gp - b) ** 2 + 4 * gp * bt).sqrt()) * 0.5 / V[0]).sqrt()


def _speeds(L, R, D, d):
    cl, cr = _fast(L, D, d), _fast(R, D, d)
    return torch.minimum(L[1 + d] - cl, R[1 + d] - cr), torch.maximum(L[1 + d] + cl, R[1 + d] + cr)


def _hll(L, R, D, d):
    sl, sr = _speeds(L, R, D, d)
    UL, UR = _cons(L, D), _cons(R, D)
    FL, FR = _flux(L, UL, D, d), _flux(R, UR, D, d)
    F = [torch.where(sl > 0, a, torch.where(sr < 0, b, (sl * sr * (v - u) + sr * a - sl * b) / (sr - sl)))
         for a, b, u, v in zip(FL, FR, UL, UR)]
    return F, torch.maximum(sl.abs(), sr.abs())


def _hlld(L, R, D, d):
    sl, sr = _speeds(L, R, D, d)
    tr = [c for c in range(D) if c != d]
    B0 = D + 2
    US, FS, S = [], [], [sl, sr]
    pts, du = [], []
    for V, s in ((L, sl), (R, sr)):
        U = _cons(V, D)
        US.append(U)
        FS.append(_flux(V, U, D, d))
        pts.append(V[D + 1] + 0.5 * sum(V[B0 + c] ** 2 for c in range(D)))
        du.append(s - V[1 + d])
    Bx = (sr * R[B0 + d] - sl * L[B0 + d]) / (sr - sl)
    sgn = torch.where(Bx > 0, 1.0, -1.0).to(F64)
    den = du[1] * R[0] - du[0] * L[0]
    SM = (du[1] * US[1][1 + d] - du[0] * US[0][1 + d] - pts[1] + pts[0]) / den
    ps = (du[1] * R[0] * pts[0] - du[0] * L[0] * pts[1] + L[0] * R[0] * du[1] * du[0] * (R[1 + d] - L[1 + d])) / den
    rs = [US[k][0] * du[k] / (S[k] - SM) for k in (0, 1)]
    sq = [r.sqrt() for r in rs]
    S1 = [SM - Bx.abs() / sq[0], SM + Bx.abs() / sq[1]]
    rev = ((S1[0] - sl) < 1e-4 * (SM - sl)) | ((S1[1] - sr) > -1e-4 * (sr - SM))
    hll = lambda n: (sr * US[1][n] - sl * US[0][n] + FS[0][n] - FS[1][n]) / (sr - sl)  # noqa: E731
    bn = torch.where(rev, (sr * US[1][B0 + d] - sl * US[0][B0 + d]) / (sr - sl), Bx)
    S1 = [torch.where(rev, SM, s) for s in S1]
    bs, vs = [], []
    for k, V in ((0, L), (1, R)):
        U = US[k]
        x = (U[0] * du[k] ** 2 - Bx ** 2) / (U[0] * du[k] * (S[k] - SM) - Bx ** 2)
        bs.append({c: torch.where(rev, hll(B0 + c), U[B0 + c] * x) for c in tr})
        vs.append({c: V[1 + c] - Bx / (U[0] * du[k]) * (bs[k][c] - U[B0 + c]) for c in tr})
    out = []
    for k, V in ((0, L), (1, R)):  # single- and double-star fluxes of side k
        U = US[k]
        us = [None] * (2 * D + 2)
        us[0], us[1 + d], us[B0 + d] = rs[k], rs[k] * SM, bn
        for c in tr:
            us[1 + c], us[B0 + c] = rs[k] * vs[k][c], bs[k][c]
        a = V[1 + d] * Bx + sum(V[1 + c] * U[B0 + c] for c in tr)
        b = SM * Bx + sum(vs[k][c] * bs[k][c] for c in tr)
        us[D + 1] = (du[k] * U[D + 1] - pts[k] * V[1 + d] + ps * SM + Bx * (a - b)) / (S[k] - SM)
        uss = list(us)
        uss[B0 + d] = Bx
        w = sq[0] + sq[1]
        vv = {c: (sq[0] * vs[0][c] + sq[1] * vs[1][c] + (bs[1][c] - bs[0][c]) * sgn) / w for c in tr}
        bb = {c: (sq[0] * bs[1][c] + sq[1] * bs[0][c] + sq[0] * sq[1] * (vs[1][c] - vs[0][c]) * sgn) / w for c in tr}
        for c in tr:
            uss[1 + c], uss[B0 + c] = rs[k] * vv[c], bb[c]
        b2 = SM * Bx + sum(vv[c] * bb[c] for c in tr)
        uss[D + 1] = us[D + 1] + (-1.0 if k == 0 else 1.0) * sgn * sq[k] * (b - b2)
        f1 = [f + S[k] * (x - u) for f, x, u in zip(FS[k], us, U)]
        f2 = [f + S1[k] * (y - x) for f, y, x in zip(f1, uss, us)]
        out.append((f1, f2))
    F = []
    for n in range(2 * D + 2):
        left = torch.where(S1[0] >= 0, out[0][0][n], out[0][1][n])
        right = torch.where(S1[1] <= 0, out[1][0][n], out[1][1][n])
        use_left = (S1[0] >= 0) | (~(S1[1] <= 0) & (SM >= 0))
        star = torch.where(use_left, left, right)
        F.append(torch.where(sl > 0, FS[0][n], torch.where(sr < 0, FS[1][n], star)))
    return F, torch.maximum(sl.abs(), sr.abs())


def _roe(L, R, D, d):
    tr = [c for c in range(D) if c != d]
    N, B0, P = 2 * D + 2, D + 2, D + 1
    g1 = GAMMA - 1
    UL, UR = _cons(L, D), _cons(R, D)
    FL, FR = _flux(L, UL, D, d), _flux(R, UR, D, d)
    dV, dU = [b - a for a, b in zip(L, R)], [b - a for a, b in zip(UL, UR)]
    ql, qr = L[0].sqrt(), R[0].sqrt()
    a_l, a_r = ql / (ql + qr), qr / (ql + qr)
    rho = a_r * L[0] + a_l * R[0]
    sr_ = rho.sqrt()
    v = [a_l * L[1 + c] + a_r * R[1 + c] for c in range(D)]
    B = [a_r * L[B0 + c] + a_l * R[B0 + c] for c in range(D)]
    u, sB = v[d], torch.where(B[d] >= 0, 1.0, -1.0).to(F64)
    b = [x / sr_ for x in B]
    bt2 = sum(b[c] ** 2 for c in tr)
    b2 = b[d] ** 2 + bt2
    bt = (bt2 * rho).sqrt()
    X = sum(dV[B0 + c] ** 2 for c in range(D)) / ((ql + qr) ** 2 * 2)
    v2 = sum(x * x for x in v)
    dp = g1 * ((0.5 * v2 - X) * dV[0] - sum(v[c] * dU[1 + c] for c in range(D)) + dU[P]
               - sum(B[c] * dU[B0 + c] for c in range(D)))
    H = sum(w * (U[P] + V[P] + 0.5 * sum(V[B0 + c] ** 2 for c in range(D))) / V[0]
            for w, U, V in ((a_l, UL, L), (a_r, UR, R)))
    Hg = H - b2
    a2 = (2 - GAMMA) * X + g1 * (Hg - 0.5 * v2)
    ca2 = b[d] ** 2
    cf2 = 0.5 * (a2 + b2 + ((a2 - b2) ** 2 + 4 * bt2 * a2).sqrt())
    cs2 = a2 * ca2 / cf2
    cf, cs, ca, a = cf2.sqrt(), cs2.sqrt(), ca2.sqrt(), a2.sqrt()
    z, one = torch.zeros_like(a), torch.ones_like(a)
    den = torch.where(cf2 != cs2, cf2 - cs2, one)
    af = ((a2 - cs2) / den).clamp(min=0).sqrt()
    as_ = ((cf2 - a2) / den).clamp(min=0).sqrt()
    slow = a <= cs
    fast = (cf == cs) | (~slow & (cf <= a))
    af = torch.where(fast, one, torch.where(slow, z, af))
    as_ = torch.where(fast, z, torch.where(slow & ~(cf == cs), one, as_))
    has = bt > 1e-9
    safe = torch.where(has, bt, one)
    if D == 2:
        be = {tr[0]: torch.where(has, torch.where(B[tr[0]] >= 0, one, -one), one)}
    else:
        be = {c: torch.where(has, B[c] / safe, one) for c in tr}
    dot = lambda w: sum(be[c] * w(c) for c in tr)  # noqa: E731
    bdv, bdB, bv = dot(lambda c: dV[1 + c]), dot(lambda c: dV[B0 + c]), dot(lambda c: v[c])
    base = X * dV[0] + dp
    waves = []  # (speed, strength, right vector)
    for sg in (-1, 1):
        for al, c_, ot, oc, sw in ((af, cf, as_, cs, 1.0), (as_, cs, af, cf, -1.0)):
            k = ot * oc * sB * sw  # fast waves carry +as cs, slow ones -af cf
            r = [None] * N
            lam = u + sg * c_
            r[0], r[1 + d], r[B0 + d] = al, al * lam, z
            for c in tr:
                r[1 + c] = al * v[c] - sg * k * be[c]
                r[B0 + c] = sw * ot * a * be[c] / sr_
            r[P] = al * (Hg + sg * u * c_) - sg * k * bv + sw * ot * a * bt / sr_
            eta = (al * base - sg * rho * k * bdv + sg * rho * al * c_ * dV[1 + d] + sw * sr_ * ot * a * bdB) * 0.5 / a2
            waves.append((lam, eta, r, True))
    r = [None] * N
    r[0], r[P] = one, 0.5 * v2 + (GAMMA - 2) / g1 * X
    for c in range(D):
        r[1 + c], r[B0 + c] = v[c], z
    waves.append((u, ((a2 - X) * dV[0] - dp) / a2, r, False))
    if D == 3:
        y, w = tr
        for sg in (-1, 1):
            r = [z] * N
            r[1 + y], r[1 + w] = sg * rho * be[w], -sg * rho * be[y]
            r[B0 + y], r[B0 + w] = -sB * sr_ * be[w], sB * sr_ * be[y]
            r[P] = sg * rho * (v[y] * be[w] - v[w] * be[y])
            eta = 0.5 * (-sg * (be[y] * dV[1 + w] - be[w] * dV[1 + y])
                         + sB / sr_ * (be[y] * dV[B0 + w] - be[w] * dV[B0 + y]))
            waves.append((u + sg * ca, eta, r, False))
    F = []
    for n in range(N):
        s = z
        for lam, eta, r, fix in waves:
            la = lam.abs()
            if fix:
                la = torch.where(la < 0.5e-6, lam * lam / 1e-6 + 0.25e-6, la)
            s = s + la * eta * r[n]
        F.append(0.5 * (FL[n] + FR[n] - s))
    return F, u.abs() + cf


_SOLVERS = {"hlld": _hlld, "hll": _hll, "roe": _roe}


def _rot(r, d):
    """variable of the rotated frame (sweep direction first) -> solver variable"""
    if r in (0, 4):
        return r
    base = 1 if r < 4 else 5
    return base + (d + r - base) % 3


def _net_layers(params):
    p = torch.as_tensor(params, dtype=F64, device=DEVICE)
    o = np.cumsum([0, NIN * NH, NH, NH * NH, NH, NH * NOUT, NOUT])
    c = [p[o[i]:o[i + 1]] for i in range(6)]
    return c[0].view(NIN, NH), c[1], c[2].view(NH, NH), c[3], c[4].view(NH, NOUT), c[5]


def _features(at, dtype=F64):
    """stencil features [.., 216] of at(rotated variable, o0, o1, o2)"""
    cen = [at(r, 0, 0, 0) for r in range(8)]
    cs = (GAMMA * cen[4] / cen[0]).sqrt()
    sb = cen[0].sqrt() * cs
    cols = []
    for r in range(8):
        for o2 in (-1, 0, 1):
            for o1 in (-1, 0, 1):
                for o0 in (-1, 0, 1):
                    s = at(r, o0, o1, o2)
                    cols.append(s / cen[r] - 1 if r in (0, 4) else (s - cen[r]) / cs if r < 4 else s / sb)
    return torch.stack(cols, -1), [cen[0], cs, cs, cs, cen[4], sb, sb, sb]


def _mlp(X, layers):
    W1, b1, W2, b2, W3, b3 = layers
    h = torch.nn.functional.silu(X @ W1 + b1)
    return torch.nn.functional.silu(h @ W2 + b2) @ W3 + b3


def _correct(V, d, g, n, states, layers):
    """the network's correction of the PLM states of the cells beg - 1 .. end along d; transversely the
    active cells and one more on each side, elsewhere the PLM states stay (they are not used)"""
    others = [q for q in range(3) if q != d]
    lo = {d: g - 1, others[0]: g - 1, others[1]: g - 1}
    m = {q: n[q] + 2 for q in range(3)}

    def at(r, o0, o1, o2):
        off = {d: o0, (d + 1) % 3: o1, (d + 2) % 3: o2}
        a = V[_rot(r, d)]
        for q in range(3):
            a = _sl(a, q, lo[q] + off[q], lo[q] + off[q] + m[q])
        return a

    X, sc = _features(at)
    shape = X.shape[:-1]
    Y = _mlp(X.reshape(-1, NIN), layers).view(*shape, NOUT)
    fall = (X.abs() > RANGE).any(-1)
    box = (slice(g - 1, g - 1 + m[2]), slice(g - 1, g - 1 + m[1]), slice(g - 1, g - 1 + m[0]))
    box = tuple(slice(None) if 2 - q == d else box[q] for q in range(3))
    new = {}
    for f in (0, 1):
        for r in range(8):
            st = states[f][_rot(r, d)][box]
            new[f, r] = st if r == 5 else st + Y[..., 8 * f + r] * sc[r]
            if r in (0, 4):
                fall = fall | ~(new[f, r] > 0)
    for (f, r), st in new.items():
        a = states[f][_rot(r, d)]
        a[box] = torch.where(fall, a[box], st)


def _ghost_index(n, g, extra):
    i = torch.arange(n + 2 * g + extra, device=DEVICE)
    w = g + (i + g * (n - 1)) % n
    return torch.where((i < g) | (i > g + n - 1 + extra), w, i)


def _fill_periodic(V, Vs, D, n, g):
    ix = [_ghost_index(n[d], g, 0) if d < D else torch.zeros(1, dtype=torch.long, device=DEVICE) for d in range(3)]
    for q in range(D + 2):
        V[q] = V[q][ix[2][:, None, None], ix[1][None, :, None], ix[0][None, None, :]]
    for c in range(D):
        jx = [_ghost_index(n[d], g, 1) if d == c else ix[d] for d in range(3)]
        Vs[c][:len(jx[2]), :len(jx[1]), :len(jx[0])] = Vs[c][jx[2][:, None, None], jx[1][None, :, None],
                                                            jx[0][None, None, :]]


def _fill_outflow(V, Vs, D, n, g, dx):
    for d in range(D):
        for side in (0, 1):
            src = g + side * (n[d] - 1)
            lo = (0, g + n[d])[side]
            for q in range(D + 2):
                a = _sl(V[q], d, src, src + 1)
                if q == 1 + d:
                    a = torch.where((1 - 2 * side) * a >= 0, torch.zeros_like(a), a)
                _sl(V[q], d, lo, lo + g).copy_(a.expand_as(_sl(V[q], d, lo, lo + g)))
            for c in range(D):
                if c == d:
                    continue
                f = Vs[c]
                for q in range(D):  # the array without its padding
                    f = _sl(f, q, 0, n[q] + 2 * g + (1 if q == c else 0))
                _sl(f, d, lo, lo + g).copy_(_sl(f, d, src, src + 1).expand_as(_sl(f, d, lo, lo + g)))
        area = [math.prod(dx[q] for q in range(D) if q != c) for c in range(D)]

        nt = [n[q] + 2 * g for q in range(D)]

        def div_other(pos):  # transverse part of div B of the cells at position pos along d
            t = 0.0
            for c in range(D):
                if c == d:
                    continue
                a = _sl(Vs[c], d, pos, pos + 1)
                for q in range(D):
                    if q not in (c, d):
                        a = _sl(a, q, 0, nt[q])
                t = t + area[c] * (_sl(a, c, 1, nt[c] + 1) - _sl(a, c, 0, nt[c]))
            return t

        normal = Vs[d]
        for q in range(D):
            if q != d:
                normal = _sl(normal, q, 0, nt[q])
        for i in range(g - 1, -1, -1):
            _sl(normal, d, i, i + 1).copy_(_sl(normal, d, i + 1, i + 2) + div_other(i) / area[d])
        for i in range(g + n[d], nt[d]):
            _sl(normal, d, i + 1, i + 2).copy_(_sl(normal, d, i, i + 1) - div_other(i) / area[d])


def _edge(a, d1, d2, o1, o2, lo, m):
    """array a at the edges lo .. lo + m, shifted by o1 along d1 and o2 along d2"""
    for q in range(3):
        if m[q] > 1 or lo[q] > 0:
            o = (o1 if q == d1 else 0) + (o2 if q == d2 else 0)
            a = _sl(a, q, lo[q] + o, lo[q] + o + m[q])
    return a


def _corner(case, e1, e2, sv1, sv2, Ec, d1, d2, lo, m):
    """corner EMF of the edges along the third direction, from the face EMFs e1 (faces normal to d1) and e2
    (normal to d2), their upwind weights and the cell EMF"""
    at = lambda a, o1, o2: _edge(a, d1, d2, o1, o2, lo, m)  # noqa: E731
    base = at(e1, 0, 0) + at(e1, 0, -1) + at(e2, 0, 0) + at(e2, -1, 0)
    if case["emf"] == "arithmetic":
        return 0.25 * base
    up = lambda w, a, b: (1 - w) * a + w * b  # noqa: E731
    for o2 in (-1, 0):  # across d1 faces: the e2 differences either side
        base = base + up(at(sv1, 0, o2), at(e2, 0, 0) - at(Ec, 0, o2), at(e2, -1, 0) - at(Ec, -1, o2))
    for o1 in (-1, 0):
        base = base + up(at(sv2, o1, 0), at(e1, 0, 0) - at(Ec, o1, 0), at(e1, 0, -1) - at(Ec, o1, -1))
    return 0.25 * base


def _advance(case, Vc, Vs, cycles, layers=None):
    """the state after some cycles, with ghosts as the last stage found them, and (t, dt)"""
    D, g = case["dims"], _ng(case)
    n = [case["nx"], case["ny"], case["nz"]]
    dx = _domain(case)
    nv = 2 * D + 2
    V = [Vc[q].clone() for q in range(nv)]
    Vs = [Vs[c].clone() for c in range(D)]
    dV = math.prod(dx[:D])
    area = [math.prod(dx[q] for q in range(D) if q != c) for c in range(D)]
    nt = [n[d] + 2 * g if d < D else 1 for d in range(3)]
    act = tuple(slice(g, g + n[d]) if d < D else slice(0, 1) for d in (2, 1, 0))
    weights = {1: [], 2: [(0.5, 0.5)], 3: [(0.25, 0.75), (2 / 3, 1 / 3)]}[case["nstages"]]
    t, dt = 0.0, _dt0(case)
    lo = [g if d < D else 0 for d in range(3)]
    m = [n[d] + 1 if d < D else 1 for d in range(3)]
    order = "plm" if case["order"] == "learned" else case["order"]
    Vs0 = U0 = None
    for cyc in range(cycles):
        for stage in range(case["nstages"]):
            if case["walls"] == "periodic":
                _fill_periodic(V, Vs, D, n, g)
            else:
                _fill_outflow(V, Vs, D, n, g, dx)
            for c in range(D):
                f = Vs[c][:nt[2] + (c == 2), :nt[1] + (c == 1), :nt[0] + (c == 0)]
                V[D + 2 + c] = 0.5 * (_sl(f, c, 0, nt[c]) + _sl(f, c, 1, nt[c] + 1))
            U = [a[act].clone() for a in _cons(V, D)]
            if stage == 0:
                U0, Vs0, inv = list(U), [a.clone() for a in Vs], 0.0
            cr = lambda a, b: V[1 + b] * V[D + 2 + a] - V[1 + a] * V[D + 2 + b]  # noqa: E731  -(v x B)_c, c = a x b
            face, upw = {}, {}
            acc = None
            for d in range(D):
                beg, end = g, g + n[d]
                st = [_recon(order, V[q], d, beg, end, dx[d], q in (0, D + 1)) for q in range(nv)]
                vl, vr = [s[0] for s in st], [s[1] for s in st]
                if layers is not None:
                    _correct(V, d, g, n, (vl, vr), layers)
                bn = Vs[d][:nt[2] + (d == 2), :nt[1] + (d == 1), :nt[0] + (d == 0)]
                bn = _sl(bn, d, beg, end + 1)
                L = [_sl(a, d, 0, n[d] + 1) for a in vr]
                R = [_sl(a, d, 1, n[d] + 2) for a in vl]
                L[D + 2 + d] = R[D + 2 + d] = bn
                F, cmax = _SOLVERS[case["solver"]](L, R, D, d)
                full = lambda x: _placed(x, d, beg, nt)  # noqa: E731
                w = torch.where(F[0] > 1e-6, 1.0, torch.where(F[0] < -1e-6, 0.0, 0.5)).to(F64)
                upw[d] = full(w)
                for c in range(D):  # E = -v x B: faces normal to d carry -+ F[B_c]
                    if c != d:
                        third = 3 - d - c
                        sg = -1.0 if (d, c) in ((0, 1), (1, 2), (2, 0)) else 1.0
                        face[d, third] = full(sg * F[D + 2 + c])
                cut = [slice(None)] * 3
                for q in range(D):
                    if q != d:
                        cut[2 - q] = slice(g, g + n[q])
                for q in range(D + 2):
                    f = F[q][tuple(cut)]
                    U[q] = U[q] - dt / dV * area[d] * (_sl(f, d, 1, n[d] + 1) - _sl(f, d, 0, n[d]))
                if stage == 0:
                    cm = cmax[tuple(cut)]
                    c = 0.5 * (_sl(cm, d, 1, n[d] + 1) + _sl(cm, d, 0, n[d])) / dx[d]
                    acc = c if acc is None else acc + c
                del st, vl, vr, L, R, F
            if stage == 0:
                inv = float(acc.max())
            E = {}
            for third, d1, d2 in ((2, 0, 1), (0, 1, 2), (1, 0, 2)):
                if D == 2 and third != 2:
                    continue
                Ec = cr(d1, d2) if third != 1 else cr(d2, d1)
                E[third] = _corner(case, face[d1, third], face[d2, third], upw[d1], upw[d2], Ec, d1, d2, lo, m)
            wc, w0 = weights[stage - 1] if stage > 0 else (1.0, 0.0)
            for c in range(D):
                s = 0.0
                for q in range(D):  # dB_c/dt = -(curl E)_c
                    if q == c:
                        continue
                    third = 3 - c - q
                    sg = 1.0 if (c, q) in ((0, 1), (1, 2), (2, 0)) else -1.0
                    e = E[third]
                    for z in range(D):
                        if z != q and z != c:
                            e = _sl(e, z, 0, n[z])
                    s = s - sg * dt / dx[q] * (_sl(e, q, 1, n[q] + 1) - _sl(e, q, 0, n[q]))
                r = tuple(slice(lo[z], lo[z] + (m[z] if z == c else n[z])) for z in (2, 1, 0))
                b = Vs[c][r] + s
                Vs[c][r] = wc * b + w0 * Vs0[c][r] if stage > 0 else b
            if stage > 0:
                U = [wc * a + w0 * b if q < D + 2 else a for q, (a, b) in enumerate(zip(U, U0))]
            Bc = []
            for c in range(D):
                f = Vs[c][tuple(slice(lo[z], lo[z] + (m[z] if z == c else n[z])) for z in (2, 1, 0))]
                Bc.append(0.5 * (_sl(f, c, 0, n[c]) + _sl(f, c, 1, n[c] + 1)))
            m2, b2 = sum(U[1 + c] ** 2 for c in range(D)), sum(x * x for x in Bc)
            p = (U[D + 1] - 0.5 * m2 / U[0] - 0.5 * b2) * (GAMMA - 1)
            V[0][act] = U[0]
            for c in range(D):
                V[1 + c][act], V[D + 2 + c][act] = U[1 + c] / U[0], Bc[c]
            V[D + 1][act] = torch.where(p <= 0, torch.full_like(p, 1e-5), p)
        t += dt
        new = case["cfl"] / inv
        dt = 1.1 * dt if new > 1.1 * dt else new
    return torch.stack(V), torch.stack(Vs), np.array([t, dt])


def _placed(x, d, beg, nt):
    """face values of the faces beg .. along d, in an array over every cell"""
    a = torch.zeros((nt[2], nt[1], nt[0]), dtype=F64, device=DEVICE)
    _sl(a, d, beg, beg + x.shape[2 - d]).copy_(x)
    return a


def _loss_grad(X, T, layers, w):
    for a in layers:
        a.requires_grad_(True)
    keep = torch.ones(NOUT, dtype=F64, device=DEVICE)
    keep[5] = keep[13] = 0.0  # the normal field components
    loss = (((_mlp(X, layers) - T) * keep).square().sum(-1)).mean() * w
    return loss, torch.cat([a.reshape(-1) for a in torch.autograd.grad(loss, layers)])


def _mix64(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9e3779b97f4a7c15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
        return z ^ (z >> np.uint64(31))


def _exact_batch(P, T, seed, base, B):
    """the batch that the counter-based sampling of the trainer picks, unrounded"""
    S, nc = P.shape[0], P.shape[2]
    h = _mix64(np.uint64(seed) ^ _mix64(np.arange(base, base + B, dtype=np.uint64)))
    dev = lambda a: torch.as_tensor(a.astype(np.int64), device=DEVICE)  # noqa: E731
    snap, cell, dire = dev(h % np.uint64(S)), dev((h >> np.uint64(16)) % np.uint64(nc ** 3)), dev(
        (h >> np.uint64(48)) % np.uint64(3))
    X = torch.empty((B, NIN), dtype=F64, device=DEVICE)
    Y = torch.empty((B, NOUT), dtype=F64, device=DEVICE)
    for d in range(3):
        s = (dire == d).nonzero().view(-1)
        q = [cell[s] % nc, cell[s] // nc % nc, cell[s] // (nc * nc)]

        def at(r, o0, o1, o2):
            p = list(q)
            for a, o in ((d, o0), ((d + 1) % 3, o1), ((d + 2) % 3, o2)):
                p[a] = (p[a] + o) % nc
            return P[snap[s], _rot(r, d), p[2], p[1], p[0]].double()

        X[s], sc = _features(at)
        for r in range(8):
            w = [at(r, o, 0, 0) for o in (-1, 0, 1)]
            hd = 0.5 * _minmod0(w[2] - w[1], w[1] - w[0])
            Y[s, r] = (T[snap[s], d, r, cell[s]].double() - (w[1] - hd)) / sc[r]
            Y[s, 8 + r] = (T[snap[s], d, 8 + r, cell[s]].double() - (w[1] + hd)) / sc[r]
    return X, Y


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        X, T = _batch(case, seed)
        loss, g = _loss_grad(X[:, :NIN].double(), T.double(), _net_layers(_params(seed)), 1.0)
        return {"grad": g, "loss": np.float64(float(loss))}
    if kind == "train":
        P, T = _dataset(case, seed)
        p = torch.as_tensor(_params(seed), dtype=F64, device=DEVICE)
        mo, ve = torch.zeros_like(p), torch.zeros_like(p)
        losses, lo, hi = [], None, None
        for s in range(case["steps"]):
            X, Y = _exact_batch(P, T, int(seed), s * case["batch"], case["batch"])
            lo = X.amin(0) if lo is None else torch.minimum(lo, X.amin(0))
            hi = X.amax(0) if hi is None else torch.maximum(hi, X.amax(0))
            loss, g = _loss_grad(X, Y, [a.clone() for a in _net_layers(p)], 1.0)
            losses.append(float(loss))
            mo, ve = 0.9 * mo + 0.1 * g, 0.999 * ve + 0.001 * g * g
            frac = s / (case["steps"] - 1) if case["steps"] > 1 else 1.0
            lr = 2e-5 + 0.5 * (2e-3 - 2e-5) * (1 + math.cos(math.pi * frac))
            p = p - lr * (mo / (1 - 0.9 ** (s + 1))) / ((ve / (1 - 0.999 ** (s + 1))).sqrt() + 1e-8)
        return {"params": p, "losses": np.array(losses), "lo": lo, "hi": hi}
    if kind == "ensemble":
        a, b = [], []
        for c, mach, beta in _ensemble_boxes(case, seed):
            Vc, Vs, _ = _advance(c, *_vortex(c, mach, beta, 0.0, 0.0), case["cycles"])
            a.append(Vc.reshape(-1))
            b.append(Vs.reshape(-1))
        return {"Vc": torch.cat(a), "Vs": torch.cat(b)}
    layers = _net_layers(_params(seed)) if kind == "learned" else None
    Vc, Vs, time = _advance(case, *_initial(case, seed), case["cycles"], layers)
    return {"Vc": Vc, "Vs": Vs, "time": time}
