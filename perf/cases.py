"""Workloads of the probe-particle AFM path, from single stages to whole fitting steps.

listed() names the workloads, draw() gives more of the same ranges, prepare() makes what a program
holds before the call, run() is one pass through the public entry points, work() the bytes and
operations a pass cannot do without, tolerance() how far another correct implementation at the
same precision may be off, exact() the same outputs from 64-bit torch code that uses none of the
package's kernels.

Sizes are those of the synthetic workloads of spammm_b200.synthetic, bench.py and the tests: 12 to
1200 atoms, grids of 64^3 to 480 x 480 x 240 nodes, rasters of 16^2 to 480^2 pixels, 12 to 60
z-steps, batches of 2 to 64 molecules.

Kinds:
  grid     force-grid build (gpu.grid_build), LJ or Morse, on-node charge or two offset charges
  scan     FIRE relaxation of a raster of z-strokes on a given grid (gpu.relax_strokes)
  df       amplitude-averaged frequency shift of an FE volume (gpu.df_amp_dir)
  image    one image through the drop-in API with NumPy arrays in and out (AFMulator)
  grad     differentiable grid path: forward, df loss and gradients (diff.GridAFM)
  direct   differentiable grid-free Morse path: forward, df loss and gradients (diff.DirectMorseAFM)
  forward  images of a batch of molecules (batch.AFMBatch.forward)
  fit      one Adam step of a batch: forward, loss, adjoint, update (batch.BatchAdam.step)
"""
import math

import numpy as np
import torch

from spammm_b200 import AFM, _lib, gpu, synthetic
from spammm_b200.AFM_utils import _lj_atoms_from_Z, _morse_atoms_from_Z
from spammm_b200.batch import AFMBatch, BatchAdam
from spammm_b200.diff import DirectMorseAFM, DirectScanSpec, GridAFM, GridScanSpec

F32, F64 = torch.float32, torch.float64
COULOMB = 14.3996448915
R2SAFE = 1e-4
STEP = 0.1                                            # node spacing and z-step (A)
ON_SITE = ([-0.05, 0, 0, 0], [0, 0, 0, 0])            # one charge at the probe position
OFF_SITES = ([0, -0.1, 0.1, 0], [0, 1.8, 3.6, 0])     # the AFMulator's default pair of offset charges


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the 38-atom molecule's 20 A cube at 0.1 A: the force grid of an everyday single image
        dict(name="grid_small", kind="grid", law="lj", atoms=38, nx=200, ny=200, nz=200, offset=False),
        # a molecule on a 3-layer NaCl slab, 48 x 48 x 24 A at 0.1 A: the largest force grid
        dict(name="grid_large", kind="grid", law="lj", atoms=1200, nx=480, ny=480, nz=240, offset=False),
        # Morse law with the default pair of offset tip charges on an odd-sized box
        dict(name="grid_morse_odd", kind="grid", law="morse", atoms=57, nx=187, ny=203, nz=149, offset=True),
        # 100 x 100 pixels x 40 z-steps over the small molecule: one everyday scan
        dict(name="scan_small", kind="scan", atoms=38, npx=100, npy=100, nz=40, zend=5.1),
        # 480 x 480 pixels x 60 z-steps over the slab: the largest single scan
        dict(name="scan_large", kind="scan", atoms=1200, npx=480, npy=480, nz=60, zend=3.1),
        # df of that scan at every height, oscillation along z
        dict(name="df_large", kind="df", nx=480, ny=480, nz=60, double=False, tilt=0.0, amp=1.0),
        # df of a small odd-sized volume with a tilted oscillation, double precision in
        dict(name="df_tilted", kind="df", nx=101, ny=97, nz=41, double=True, tilt=0.2, amp=0.5),
        # the smallest whole call: a tiny image through the drop-in API, where latency counts
        dict(name="image_tiny", kind="image", atoms=14, ngrid=64, npx=24, nz=20),
        # gradients of a df loss on the small molecule, one image per step of a user's own optimiser
        dict(name="grad_image", kind="grad", law="lj", atoms=38, ngrid=200, npx=100, npy=100, nz=40, zend=5.1),
        # the same through the grid-free Morse path
        dict(name="direct_image", kind="direct", atoms=38, npx=100, npy=100, nz=40),
        # images of 64 molecules of uneven sizes, grid slabs + relaxation + df
        dict(name="forward_batch", kind="forward", mols=64, set=3, natoms=120, npx=256, nz=60),
        # one fitting step of 64 molecules on positions and charges
        dict(name="fit_batch", kind="fit", mols=64, set=5, natoms=120, npx=256, nz=60),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["grid", "grid", "scan", "df", "image", "grad", "direct", "forward", "fit"])
    if kind == "grid":
        c = dict(kind=kind, law=rng.choice(["lj", "morse"]), atoms=log(12, 1200), nx=log(64, 480), ny=log(64, 480),
                 nz=log(64, 240), offset=rng.random() < 0.4)
        cost = c["atoms"] * c["nx"] * c["ny"] * c["nz"] * (2.5 if c["law"] == "morse" or c["offset"] else 1.0)
        if cost > 1200 * 480 * 480 * 240:  # the costlier laws on fewer atoms
            c["atoms"] = max(12, int(c["atoms"] * 1200 * 480 * 480 * 240 / cost))
        return c
    if kind == "scan":
        return dict(kind=kind, atoms=log(12, 120), npx=log(16, 480), npy=log(16, 480), nz=rng.randint(12, 60),
                    zend=round(rng.uniform(4.0, 6.1), 1))
    if kind == "df":
        tilt = rng.choice([0.0, 0.0, 0.2])
        top = 480 if tilt == 0.0 else 128
        return dict(kind=kind, nx=log(16, top), ny=log(16, top), nz=rng.randint(12, 60), double=rng.random() < 0.3,
                    tilt=tilt, amp=round(rng.uniform(0.3, 1.5), 2))
    if kind == "image":
        return dict(kind=kind, atoms=log(12, 120), ngrid=log(64, 200), npx=log(16, 128), nz=rng.randint(12, 40))
    if kind == "grad":
        return dict(kind=kind, law=rng.choice(["lj", "morse"]), atoms=log(12, 120), ngrid=log(140, 240),
                    npx=log(16, 128), npy=log(16, 128), nz=rng.randint(12, 40), zend=round(rng.uniform(4.5, 6.0), 1))
    if kind == "direct":
        return dict(kind=kind, atoms=log(12, 120), npx=log(16, 128), npy=log(16, 128), nz=rng.randint(12, 40))
    return dict(kind=kind, mols=log(2, 48), set=rng.randint(10, 10 ** 6), natoms=rng.randint(20, 120),
                npx=rng.randint(65, 256), nz=rng.randint(31, 60))


# ------------------------------------------------------------------------------------------ inputs
def _system(case, seed):
    """(atoms (na,4), params) float32 NumPy: a planar C/N/O/H molecule; beyond 200 atoms on a NaCl slab
    3 A below it (ions displaced by 0.02 A).  LJ or Morse parameters from the element table."""
    na = int(case["atoms"])
    law = _morse_atoms_from_Z if case.get("law", "lj") == "morse" else _lj_atoms_from_Z
    rng = np.random.default_rng(seed)
    nm = na if na <= 200 else 60
    nh, nn, no = max(1, nm // 5), nm // 9, nm // 8
    pos, Z, q = synthetic.planar_molecule({"C": nm - nh - nn - no, "N": nn, "O": no, "H": nh}, int(seed) + 1)
    if na > nm:
        ions = na - nm
        side = int(math.ceil(math.sqrt(ions / 3.0)))
        sp, sZ, sq = synthetic.nacl_slab(side, int(math.ceil(ions / (3.0 * side))), 3)
        sp, sZ, sq = sp[:ions], sZ[:ions], sq[:ions]
        pos[:, 2] += 3.0
        pos = np.concatenate([sp + rng.normal(0.0, 0.02, sp.shape), pos])
        Z, q = np.concatenate([sZ, Z]), np.concatenate([sq, q])
    atoms, prm = law(pos, Z)
    atoms[:, 3] = q
    return atoms, prm


def _sites(case):
    Qs, QZs = OFF_SITES if case.get("offset") else ON_SITE
    return np.array(Qs, np.float32), np.array(QZs, np.float32)


def _box(case):
    """Grid origin, node counts and the vectors of grid_build: centred in x and y, 8 A (6 A for the small
    molecules' cubes) below z = 0, as the plain workloads' grids."""
    n = (case["nx"], case["ny"], case["nz"])
    o = np.array([-STEP * n[0] / 2, -STEP * n[1] / 2, -8.0 if case["atoms"] > 200 else -min(6.0, 0.3 * STEP * n[2])])
    return o, n, (np.array([*o, 0], np.float32), np.array([STEP, 0, 0, 0], np.float32),
                  np.array([0, STEP, 0, 0], np.float32), np.array([0, 0, STEP, 0], np.float32))


def _raster(npx, npy, z, span=None):
    """(npx*npy, 4) float32 tip positions, ix-major, 0.1 A pixels (or `span` A wide)."""
    d = STEP if span is None else span / max(npx, npy)
    x = (np.arange(npx) - npx / 2) * d
    y = (np.arange(npy) - npy / 2) * d
    p = np.zeros((npx * npy, 4), np.float32)
    p[:, 0], p[:, 1], p[:, 2] = np.repeat(x, npy), np.tile(y, npx), z
    return p


def _top(case):
    """Height of the outermost plane of atoms."""
    return 3.0 if case["atoms"] > 200 else 0.0


def _field(dtype, atoms, prm, Qs, QZs, X, Y, Z, cap=True):
    """(..., 4) force field at the broadcast of X, Y, Z from the pair laws, summed atom by atom."""
    dev = X.device
    A, P = torch.as_tensor(atoms).to(dev, F64).tolist(), torch.as_tensor(prm).to(dev, F64).tolist()
    shape = torch.broadcast_shapes(X.shape, Y.shape, Z.shape)
    out = torch.zeros((4,) + shape, dtype=dtype, device=dev)
    sites = [(float(q) * COULOMB, float(z)) for q, z in zip(Qs, QZs) if q != 0]
    for a, p in zip(A, P):
        dx, dy, dz = X - a[0], Y - a[1], Z - a[2]
        dxy = dx * dx + dy * dy + R2SAFE
        r2 = dxy + dz * dz
        if len(p) == 2:
            i2 = 1.0 / r2
            i6 = i2 * i2 * i2
            out[3] += (p[1] * i6 - p[0]) * i6
            s = i6.mul_(12 * p[1] * i6 - 6 * p[0]).mul_(i2)
        else:
            r = torch.sqrt(r2)
            e = torch.exp(p[2] * (r - p[0]))
            out[3] += p[1] * e * (e - 2)
            s = (-2 * p[2] * p[1]) * e * (e - 1) / r
        for q, z in sites:
            if z == 0.0:
                E = (q * a[3]) * torch.rsqrt(r2)
                out[3] += E
                s += E / r2
        out[0] += dx * s
        out[1] += dy * s
        out[2] += dz * s
        for q, z in sites:
            if z != 0.0:
                dk = dz + z
                rk = dxy + dk * dk
                E = (q * a[3]) * torch.rsqrt(rk)
                sk = E / rk
                out[3] += E
                out[0] += dx * sk
                out[1] += dy * sk
                out[2] += dk * sk
    if cap:
        over = out[3].abs() > 100.0
        out = torch.where(over, out * (100.0 / out[3].abs().clamp_min(1e-30)), out)
    return out.movedim(0, -1).contiguous()


def _axes(o, n, dtype):
    ax = [torch.as_tensor(np.float32(o[d]) + np.float32(STEP) * np.arange(n[d], dtype=np.float64), device="cuda").to(dtype)
          for d in range(3)]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _scan_grid(case, seed):
    """Grid of a scan: the band of nodes the strokes can reach, in plain torch (an input of the case)."""
    atoms, prm = _system(case, seed)
    n_xy = int(max(case["npx"], case["npy"])) + 24
    top = _top(case)
    z_end, z_top = top + case["zend"], top + case["zend"] + STEP * (case["nz"] - 1)
    n = (n_xy, n_xy, int(round((z_top - z_end) / STEP)) + 24)
    o = np.array([-STEP * n_xy / 2, -STEP * n_xy / 2, z_end - 1.2])
    return atoms, prm, o, n, z_top


def _dinv(o, n):
    L = np.array(n, np.float64) * STEP
    return [np.array([(1 / L[d] if c == d else 0.0) for c in range(3)] + [-np.float32(o[d]) / L[d] + 0.5 / n[d]],
                     np.float32) for d in range(3)]


def _volume(case, seed):
    """(nx,ny,nz,4) FE volume of a corrugated surface: LJ-like Fz(z) whose depth varies over the pixels."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z = 5.0 + STEP * torch.arange(nz, device="cuda", dtype=F64)
    depth = 0.02 * (1 + 0.5 * torch.rand((nx, ny, 1), generator=g, device="cuda", dtype=F64))
    u = (3.5 + 0.2 * torch.rand((nx, ny, 1), generator=g, device="cuda", dtype=F64)) / z
    fes = torch.empty((nx, ny, nz, 4), device="cuda", dtype=F64)
    fes[..., 2] = 12 * depth * (u ** 13 - u ** 7)
    fes[..., 3] = depth * (u ** 12 - 2 * u ** 6) * z
    fes[..., :2] = 0.2 * depth[..., None] * u[..., None] ** 7 * torch.randn((nx, ny, 1, 2), generator=g, device="cuda",
                                                                            dtype=F64)
    return fes if case["double"] else fes.to(F32)


def _target(shape, seed):
    """A target df of the size the images have (eV/A^2)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 7)
    return 0.01 * torch.randn(shape, generator=g, device="cuda", dtype=F64)


def _items(case, seed):
    """Molecules of the batch distribution (sizes from the case's set) with the seed's positions and charges."""
    items = synthetic.batch_molecules(case["mols"], seed=case["set"], natoms=(10, case["natoms"]), npx=(64, case["npx"]), nzs=(30, case["nz"]))
    rng = np.random.default_rng(seed)
    for it in items:
        it.atoms[:, :3] += rng.normal(0.0, 0.02, (len(it.atoms), 3)).astype(np.float32)
        it.atoms[:, 3] += rng.normal(0.0, 0.02, len(it.atoms)).astype(np.float32)
    return items


def _grad_spec(case):
    n = (case["ngrid"],) * 3
    o = np.array([-STEP * n[0] / 2, -STEP * n[1] / 2, -2.0 if n[0] < 200 else -6.0])
    z_top = case["zend"] + STEP * (case["nz"] - 1)
    return GridScanSpec(kind=_lib.SPM_KIND_MORSE if case["law"] == "morse" else _lib.SPM_KIND_LJ, ngrid=n, origin=o,
                        step=STEP, points=_raster(case["npx"], case["npy"], z_top, 10.0), nz=case["nz"], dtip=-STEP,
                        raster_ny=case["npy"], strict=False, polish=True)


def _direct_spec(case):
    # the probe hangs 4 A under its anchor: it starts at 9 A above the molecule
    return DirectScanSpec(points=_raster(case["npx"], case["npy"], 13.0, 10.0), nz=case["nz"], dtip=-STEP,
                          raster_ny=case["npy"], strict=False)


def _image_box(case):
    n = case["ngrid"]
    z_end = 5.0 if n >= 100 else 4.0
    return np.array([-STEP * n / 2, -STEP * n / 2, z_end + STEP * case["nz"] + 1.2 - STEP * n]), (n, n, n), z_end


def _image_raster(case):
    x = ((np.arange(case["npx"]) + 0.5) / case["npx"] - 0.5) * (0.6 * STEP * case["ngrid"])
    return x.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grid":
        atoms, prm = _system(case, seed)
        _, n, vec = _box(case)
        Qs, QZs = _sites(case)
        law = _lib.SPM_KIND_MORSE if case["law"] == "morse" else _lib.SPM_KIND_LJ
        return dict(kind=kind, args=(law, torch.as_tensor(atoms).cuda(), torch.as_tensor(prm).cuda(), n, *vec, Qs, QZs))
    if kind == "scan":
        atoms, prm, o, n, z_top = _scan_grid(case, seed)
        k, d0, Qs, QZs = synthetic.probe_params()
        grid = _field(F32, atoms, prm, Qs, QZs, *_axes(o, n, F32))
        P = _lib.make_scan_params(dinv=_dinv(o, n), dTip=[0, 0, -STEP, 0], stiffness=k, dpos0=d0,
                                  relax_params=[0.5, 0.1, 0.02, 0.5], nz=case["nz"], max_iter=1000, f2conv=1e-10,
                                  flip_z=True, raster_ny=case["npy"])
        return dict(kind=kind, grid=grid, P=P, pts=torch.as_tensor(_raster(case["npx"], case["npy"], z_top)).cuda())
    if kind == "df":
        return dict(kind=kind, fes=_volume(case, seed), dir=(case["tilt"], 0.5 * case["tilt"], 1.0), amp=case["amp"])
    if kind == "image":
        atoms, prm = _system(case, seed)
        k, d0, Qs, QZs = synthetic.probe_params()
        afm = AFM.AFMulator(use_morse=False)
        afm.n_relax_max, afm.f2conv, afm.newton_polish = 1000, 1e-10, True
        afm.tipQs, afm.tipQZs = Qs, QZs
        o, n, z_end = _image_box(case)
        return dict(kind=kind, afm=afm, atoms=atoms, prm=prm, o=o, n=n, k=k, d0=d0, xs=_image_raster(case),
                    heights=(z_end + STEP * np.arange(case["nz"])).astype(np.float32))
    if kind in ("grad", "direct"):
        atoms, prm = _system(case if kind == "grad" else dict(case, law="morse"), seed)
        s = dict(kind=kind, atoms=torch.as_tensor(atoms).cuda().requires_grad_(True),
                 prm=torch.as_tensor(prm).cuda().requires_grad_(True), shape=(case["npx"], case["npy"], case["nz"]),
                 target=_target((case["npx"], case["npy"], case["nz"]), seed))
        if kind == "direct":
            return dict(s, spec=_direct_spec(case))
        k = torch.as_tensor(synthetic.probe_params()[0]).requires_grad_(True)
        return dict(s, spec=_grad_spec(case), k=k)
    b = AFMBatch(_items(case, seed))
    if kind == "forward":
        return dict(kind=kind, batch=b)
    # the target images: the molecules with positions displaced by 0.1 A
    start = b.atoms.clone()
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 3)
    b.set_relax_options(polish=True)
    b.atoms[:, :3] += 0.1 * torch.randn((b.total_atoms, 3), generator=g, device="cuda", dtype=F32)
    b.build_grids()
    b.relax()
    b.loss_seed()
    b.set_target_states(b.df_c.clone())
    b.atoms.copy_(start)
    b.set_relax_options(warm=True)
    b.reset_warm_start()
    b.enable_failure_mask()
    return dict(kind=kind, batch=b, adam=BatchAdam(b, lr=0.01))


def run(state):
    kind = state["kind"]
    if kind == "grid":
        return gpu.grid_build(*state["args"])
    if kind == "scan":
        return gpu.relax_strokes(state["grid"], state["P"], state["pts"])
    if kind == "df":
        return gpu.df_amp_dir(state["fes"], STEP, state["dir"], state["amp"])
    if kind == "image":
        afm, n = state["afm"], state["n"]
        afm.atoms_arr, afm.cLJs_arr = state["atoms"], state["prm"]
        afm.setup_grid_world(state["o"], np.array(n) * STEP, n)
        afm.make_forcefield()
        afm.setup_fdbm_grid_from_img(afm.img_FF, n, state["o"], STEP)
        fes, disp = afm.scan_fdbm(state["xs"], state["xs"], state["heights"], mol_z=0.0, bond_length=0.0,
                                  stiffness=state["k"], dpos0=state["d0"])
        return dict(fes=fes, disp=disp, df=AFM.compute_df_amp_dir(fes, (STEP,) * 3, (0., 0., 1.), 1.0))
    if kind in ("grad", "direct"):
        a, p, spec, (nx, ny, nz) = state["atoms"], state["prm"], state["spec"], state["shape"]
        if kind == "grad":
            fes = GridAFM.apply(a, p, state["k"], spec)
        else:
            fes = DirectMorseAFM.apply(a, p, spec)
        loss, df, dL = gpu.df_loss_seed(fes.detach().view(nx, ny, nz, 4), state["target"], spec.dtip)
        wrt = (a, p, state["k"]) if kind == "grad" else (a, p)
        g = torch.autograd.grad(fes, wrt, dL.view(nx * ny, nz, 4))
        return dict(fes=fes.detach(), loss=loss, df=df, **{"grad_" + n: v for n, v in zip(("atoms", "prm", "k"), g)})
    b = state["batch"]
    if kind == "forward":
        b.forward(amp=1.0)
        return dict(fes=b.FEs, pos=b.PPs[:, :3], df=b.df)
    state["adam"].step()
    return dict(loss=b.loss, grad=b.grad, atoms=b.atoms, df=b.df_c)


# ------------------------------------------------------------------------------------------ measures
def _batch_sizes(case):
    items = synthetic.batch_molecules(case["mols"], seed=case["set"], natoms=(10, case["natoms"]),
                                      npx=(64, case["npx"]), nzs=(30, case["nz"]))
    states = sum(it.n_scan * it.nz for it in items)
    # nodes between the strokes' ends and under the raster
    nodes = [(float(it.xs[-1] - it.xs[0]) / STEP + 2) ** 2 * (it.nz + 1) for it in items]
    return states, sum(nodes), sum(n * len(it.atoms) for n, it in zip(nodes, items))


def work(case):
    """Inputs read once, outputs written once; flops of the pair sums as the laws define them (an expansion
    of distant atoms needs fewer) and of about ten evaluations of a trilinear sample per relaxed state."""
    kind = case["kind"]
    pair = 49 if case.get("law", "lj") == "lj" and not case.get("offset") else 80
    if kind == "grid":
        nodes = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=16.0 * nodes + 32.0 * case["atoms"], flops=float(pair) * nodes * case["atoms"])
    if kind == "df":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=n * ((32 if case["double"] else 16) + 4.0), flops=45.0 * n)
    if kind in ("forward", "fit"):
        states, nodes, pairs = _batch_sizes(case)
        per = 36.0 if kind == "forward" else 200.0
        return dict(bytes=16.0 * nodes + per * states, flops=49.0 * pairs + 1000.0 * states)
    states = case["npx"] * case.get("npy", case["npx"]) * case["nz"]
    sample = 1000.0 * states
    if kind == "scan":
        n = _scan_grid_nodes(case)
        return dict(bytes=16.0 * n + 32.0 * states, flops=sample)
    if kind == "direct":
        return dict(bytes=120.0 * states, flops=80.0 * 12 * case["atoms"] * states)
    nodes = case["ngrid"] ** 3
    per, passes = (36.0, 1) if kind == "image" else (120.0, 2)
    return dict(bytes=16.0 * nodes + per * states, flops=passes * 49.0 * case["atoms"] * nodes + sample)


def _scan_grid_nodes(case):
    return (max(case["npx"], case["npy"]) + 24) ** 2 * (case["nz"] + 23)


def tolerance(case):
    kind = case["kind"]
    if kind == "scan":
        # the relaxation's operation order is part of its contract (the CPU oracle repeats it): same bits
        return "exact"
    # the others: about four times what the same system with its atoms in another order gives
    if kind == "grid":
        # the norm is that of the nodes inside the atoms, where the float32 node coordinates count
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "df":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "image":
        return {"rel": 1e-4, "max": 1e-3}
    if kind == "grad":
        return {"rel": 1e-4, "max": 1e-3}
    if kind == "direct":
        # FIRE stops at |F| < 1e-4 eV/A: a step more or less moves a state by its stopping slack
        return {"rel": 1e-3, "max": 0.08}
    if kind == "forward":
        # unpolished FIRE stops at |F| < 1e-5 eV/A, up to 5e-3 A from the equilibrium
        return {"rel": 6e-4, "max": 0.05}
    # polished equilibria and their gradients, after up to three steps
    return {"rel": 1e-4, "max": 5e-3}


# ------------------------------------------------------------------------------------------ 64 bits
def _sample(grid, o, n, q):
    """Trilinear periodic sample of a (nz,ny,nx,4) FP64 grid at q (m,3): (FE (m,4), dFE/dq (m,4,3), corner
    indices (m,8), corner weights (m,8))."""
    dinv = _dinv(o, n)
    nx, ny, nz = n
    i0, w, t1 = [], [], []
    for d in range(3):
        u = q[:, d] * float(dinv[d][d]) + float(dinv[d][3])
        t = (u - torch.floor(u)) * n[d] - 0.5
        f = torch.floor(t)
        i0.append(f.to(torch.int64))
        w.append(t - f)
        t1.append(float(dinv[d][d]) * n[d])
    idx, wt, dw = [], [], []
    for k in range(2):
        for j in range(2):
            for i in range(2):
                idx.append((((i0[2] + k) % nz) * ny + (i0[1] + j) % ny) * nx + (i0[0] + i) % nx)
                c = [w[d] if b else 1 - w[d] for d, b in enumerate((i, j, k))]
                s = [1.0 if b else -1.0 for b in (i, j, k)]
                wt.append(c[0] * c[1] * c[2])
                dw.append(torch.stack([s[0] * t1[0] * c[1] * c[2], s[1] * t1[1] * c[0] * c[2], s[2] * t1[2] * c[0] * c[1]], 1))
    idx, wt, dw = torch.stack(idx, 1), torch.stack(wt, 1), torch.stack(dw, 1)
    v = grid.view(-1, 4)[idx]
    return (wt[..., None] * v).sum(1), torch.einsum("mcd,mcf->mfd", dw, v), idx, wt


def _spring(d, k, d0):
    f = (d - d0[:3]) * k[:3]
    if float(k[3]) != 0.0:
        r = d.norm(dim=1, keepdim=True)
        f = f + d * (float(k[3]) * (r - float(d0[3])) / r)
    return f


def _spring_jac(d, k, d0):
    J = torch.diag(k[:3]).expand(d.shape[0], 3, 3)
    if float(k[3]) != 0.0:
        r = d.norm(dim=1)[:, None, None]
        kw, l0 = float(k[3]), float(d0[3])
        J = J + kw * (1 - l0 / r) * torch.eye(3, device=d.device, dtype=F64) + kw * l0 / r ** 3 * d[:, :, None] * d[:, None, :]
    return J


def _fire(field, tip, nz, dtip, k, d0, max_iter, f2conv, test_first, polish=None):
    """FIRE strokes in FP64 -> per z-step (FE, position, converged).  field(q, rows) -> FE (m,4); test_first:
    the convergence test precedes the update (PP bookkeeping) and FE is the sample at the stored position,
    else the last in-loop sample.  polish(q, tip) -> the equilibrium near q (the outputs; the stroke goes on
    from the unpolished position)."""
    m, dev = tip.shape[0], tip.device
    k, d0 = (torch.as_tensor(np.asarray(v, np.float64), device=dev) for v in (k, d0))
    dt0, damp0 = 0.5, float(np.float32(0.1))
    pos = tip + d0[:3]
    dt, damp = torch.full((m, 1), dt0, device=dev, dtype=F64), torch.full((m, 1), damp0, device=dev, dtype=F64)
    out = []
    for _ in range(nz):
        v = torch.zeros_like(pos)
        fe_o = torch.zeros((m, 4), device=dev, dtype=F64)
        ok = torch.zeros(m, device=dev, dtype=torch.bool)
        live = torch.arange(m, device=dev)
        for it in range(max_iter):
            q = pos[live]
            fe = field(q, live)
            f = fe[:, :3] + _spring(q - tip[live], k, d0)
            fe_o[live] = fe
            ff = (f * f).sum(1, keepdim=True)
            done = ff[:, 0] < f2conv
            ok[live[done]] = True
            vl, dl, pl = v[live], dt[live], damp[live]
            vv, vf = (vl * vl).sum(1, keepdim=True), (vl * f).sum(1, keepdim=True)
            back = vf < 0
            cf = pl * torch.sqrt(vv / (ff + 1e-8))
            vl = torch.where(back, torch.zeros_like(vl), vl * (1 - pl) + f * cf)
            dl = torch.where(back, (dl * 0.5).clamp_min(0.1 * dt0), (dl * 1.1).clamp_max(dt0))
            pl = torch.where(back, torch.full_like(pl, damp0), pl * 0.99)
            vl = vl + f * dl
            if test_first:
                go = ~done
                v[live[go]], dt[live[go]], damp[live[go]] = vl[go], dl[go], pl[go]
                pos[live[go]] = (q + vl * dl)[go]
            else:
                v[live], dt[live], damp[live], pos[live] = vl, dl, pl, q + vl * dl
            live = live[~done]
            if live.numel() == 0:
                break
        if test_first and live.numel():
            fe_o[live] = field(pos[live], live)
        q = pos.clone()
        if polish is not None:
            q, fe_o = polish(q, tip)
        out.append((fe_o, q, ok, tip.clone()))
        tip = tip.clone()
        tip[:, 2] += dtip
        pos = pos.clone()
        pos[:, 2] += dtip
    return out


def _df_amp(fes, spacing, direction, amp):
    """The amplitude-averaged df of a volume, nine Gauss-Chebyshev nodes, in FP64."""
    n = np.asarray(direction, np.float64)
    n = n / np.linalg.norm(n)
    F = fes.to(F64)
    Fn = F[..., 0] * n[0] + F[..., 1] * n[1] + F[..., 2] * n[2]
    acc = torch.zeros_like(Fn)
    for u in np.cos((2 * np.arange(9) + 1) / 18 * np.pi):
        S = Fn
        for ax in range(3):  # linear interpolation is separable
            c = torch.arange(Fn.shape[ax], device=Fn.device, dtype=F64) + u * amp * n[ax] / spacing
            f = torch.floor(c)
            t = (c - f).reshape([-1 if d == ax else 1 for d in range(3)])
            lo = f.to(torch.int64).clamp(0, Fn.shape[ax] - 1)
            hi = (f.to(torch.int64) + 1).clamp(0, Fn.shape[ax] - 1)
            S = S.index_select(ax, lo) * (1 - t) + S.index_select(ax, hi) * t
        for ax in range(3):
            if abs(n[ax]) > 1e-15:
                acc -= n[ax] / 9 * torch.gradient(S, spacing=spacing, dim=ax)[0]
    return acc


def _strokes64(case, atoms, prm, o, n, pts, z_lo, z_hi, k, d0, nz, polish, test_first, Qs, QZs, law=None):
    """FP64 grid over the layers the strokes can reach and the FP64 relaxation on it."""
    lo, hi = max(0, int((z_lo - o[2]) / STEP) - 3), min(n[2], int((z_hi - o[2]) / STEP) + 5)
    X, Y, Z = _axes(o, n, F64)
    grid = torch.zeros((n[2], n[1], n[0], 4), device="cuda", dtype=F64)
    grid[lo:hi] = _field(F64, atoms, prm, Qs, QZs, X, Y, Z[lo:hi])
    kt = torch.as_tensor(np.asarray(k, np.float64), device="cuda")
    dt = torch.as_tensor(np.asarray(d0, np.float64), device="cuda")

    def newton(q, tip):
        for _ in range(6):
            fe, J, _, _ = _sample(grid, o, n, q)
            G = fe[:, :3] + _spring(q - tip, kt, dt)
            step = torch.linalg.solve(J[:, :3] + _spring_jac(q - tip, kt, dt), G[..., None])[..., 0]
            q1 = q - step.clamp(-0.1, 0.1)
            G1 = _sample(grid, o, n, q1)[0][:, :3] + _spring(q1 - tip, kt, dt)
            better = (G1 * G1).sum(1) < (G * G).sum(1)
            q = torch.where(better[:, None], q1, q)
        return q, _sample(grid, o, n, q)[0]

    tip = torch.as_tensor(pts[:, :3], device="cuda").to(F64)
    return grid, _fire(lambda q, rows: _sample(grid, o, n, q)[0], tip, nz, -STEP, k, d0, 1000, 1e-10, test_first,
                       newton if polish else None)


def _loss64(fes, target):
    """df, loss and dL/dFz of the central-difference df loss ((pixels, nz) in stroke order)."""
    Fz = fes[..., 2].detach().clone().requires_grad_(True)
    df = torch.zeros_like(Fz)
    df[..., 1:-1] = -(Fz[..., 2:] - Fz[..., :-2]) / (2 * STEP)
    w = torch.ones_like(Fz)
    w[..., 0] = 0
    w[..., -1] = 0
    loss = 0.5 * (w * (df - target) ** 2).sum() / w.sum()
    return loss.detach().reshape(1), df.detach(), torch.autograd.grad(loss, Fz)[0]


def _lam(J, rhs, ok):
    """J^T lambda = rhs where the state is converged and stable, 0 elsewhere; also the mask."""
    S = -0.5 * (J + J.transpose(1, 2)) - 1e-5 * torch.eye(3, device=J.device, dtype=F64)
    m2 = S[:, 0, 0] * S[:, 1, 1] - S[:, 0, 1] ** 2
    ok = ok & (S[:, 0, 0] > 0) & (m2 > 0) & (torch.linalg.det(S) > 0)  # smallest eigenvalue of -J above 1e-5
    lam = torch.linalg.solve(J.transpose(1, 2), rhs[..., None])[..., 0]
    return torch.where(ok[:, None], lam, torch.zeros_like(lam)), ok


def _exact_grad(case, seed):
    atoms, prm = _system(case, seed)
    spec = _grad_spec(case)
    k, d0, Qs, QZs = synthetic.probe_params()
    o, n, nz = spec.origin, spec.ngrid, spec.nz
    grid, st = _strokes64(case, atoms, prm, o, n, spec.points, case["zend"] - 1, float(spec.points[0, 2]) + 1, k, d0,
                          nz, True, True, Qs, QZs)
    fes = torch.stack([s[0] for s in st], 1)
    shape = (case["npx"], case["npy"], nz)
    loss, df, dFz = _loss64(fes.view(*shape, 4), _target(shape, seed))
    q, ok, tip = (torch.stack([s[i] for s in st], 1) for i in (1, 2, 3))
    q, ok, tip = q.reshape(-1, 3), ok.reshape(-1), tip.reshape(-1, 3)
    _, J, idx, wt = _sample(grid, o, n, q)
    kt = torch.as_tensor(np.asarray(k, np.float64), device="cuda")
    dt = torch.as_tensor(np.asarray(d0, np.float64), device="cuda")
    u = torch.zeros((q.shape[0], 4), device="cuda", dtype=F64)
    u[:, 2] = dFz.reshape(-1)
    lam, ok = _lam(J[:, :3] + _spring_jac(q - tip, kt, dt), torch.einsum("mf,mfd->md", u, J), ok)
    u = torch.where(ok[:, None], u, torch.zeros_like(u))
    ubar = torch.cat([u[:, :3] - lam, u[:, 3:]], 1)
    uniq, inv = torch.unique(idx.reshape(-1), return_inverse=True)
    gbar = torch.zeros((uniq.numel(), 4), device="cuda", dtype=F64)
    gbar.index_add_(0, inv, (wt[..., None] * ubar[:, None, :]).reshape(-1, 4))
    A = torch.as_tensor(atoms).cuda().to(F64).requires_grad_(True)
    P = torch.as_tensor(prm).cuda().to(F64).requires_grad_(True)
    X, Y, Z = (a.reshape(-1) for a in _axes(o, n, F64))
    nodes = torch.stack([X[uniq % n[0]], Y[(uniq // n[0]) % n[1]], Z[uniq // (n[0] * n[1])]], 1)
    gA, gP = torch.zeros_like(A), torch.zeros_like(P)
    for c in range(0, uniq.numel(), 100000):
        a, p = torch.autograd.grad((_pairs64(nodes[c:c + 100000], A, P, Qs, QZs) * gbar[c:c + 100000]).sum(), (A, P))
        gA += a
        gP += p
    d = q - tip
    dk = torch.zeros(4, device="cuda", dtype=F64)
    dk[:3] = -(lam * (d - dt[:3])).sum(0)
    dk[3] = -((lam * d).sum(1) * (d.norm(dim=1) - dt[3]) / d.norm(dim=1)).sum()
    return dict(fes=fes, loss=loss, df=df, grad_atoms=gA, grad_prm=gP, grad_k=dk)


def _pairs64(q, A, P, Qs, QZs):
    """(m, 4) field at points q as a torch function of q, atoms A and parameters P (uncapped)."""
    d = q[:, None, :] - A[None, :, :3]
    r2 = (d * d).sum(-1) + R2SAFE
    if P.shape[1] == 2:
        i2 = 1.0 / r2
        i6 = i2 ** 3
        E = (P[:, 1] * i6 - P[:, 0]) * i6
        s = (12 * P[:, 1] * i6 - 6 * P[:, 0]) * i6 * i2
    else:
        r = torch.sqrt(r2)
        e = torch.exp(P[:, 2] * (r - P[:, 0]))
        E = P[:, 1] * e * (e - 2)
        s = (-2 * P[:, 2] * P[:, 1]) * e * (e - 1) / r
    F = (d * s[..., None]).sum(1)
    E = E.sum(1)
    for c, z in zip(Qs, QZs):
        if c == 0:
            continue
        dk = d + torch.tensor([0.0, 0.0, float(z)], device=q.device, dtype=F64)
        ir = torch.rsqrt((dk * dk).sum(-1) + R2SAFE)
        Ec = float(c) * COULOMB * A[:, 3] * ir
        F = F + (dk * (Ec * ir * ir)[..., None]).sum(1)
        E = E + Ec.sum(1)
    return torch.cat([F, E[:, None]], 1)


def _exact_direct(case, seed):
    atoms, prm = _system(dict(case, law="morse"), seed)
    spec = _direct_spec(case)
    A = torch.as_tensor(atoms).cuda().to(F64).requires_grad_(True)
    P = torch.as_tensor(prm).cuda().to(F64).requires_grad_(True)
    with torch.no_grad():
        st = _fire(lambda q, rows: _pairs64(q, A, P, spec.tipQs, spec.tipQZs),
                   torch.as_tensor(spec.points[:, :3], device="cuda").to(F64), spec.nz, spec.dtip, spec.stiffness,
                   spec.dpos0, spec.max_iter, spec.f2conv, True)
    fes = torch.stack([s[0] for s in st], 1)
    shape = (case["npx"], case["npy"], spec.nz)
    loss, df, dFz = _loss64(fes.view(*shape, 4), _target(shape, seed))
    q, ok, tip = (torch.stack([s[i] for s in st], 1) for i in (1, 2, 3))
    q, ok, tip, dFz = q.reshape(-1, 3), ok.reshape(-1), tip.reshape(-1, 3), dFz.reshape(-1)
    kt = torch.as_tensor(np.asarray(spec.stiffness, np.float64), device="cuda")
    dt = torch.as_tensor(np.asarray(spec.dpos0, np.float64), device="cuda")
    gA, gP = torch.zeros_like(A), torch.zeros_like(P)
    for c in range(0, q.shape[0], 100000):
        s = slice(c, c + 100000)
        qc = q[s].clone().requires_grad_(True)
        fe = _pairs64(qc, A, P, spec.tipQs, spec.tipQZs)
        J = torch.stack([torch.autograd.grad(fe[:, f].sum(), qc, retain_graph=True)[0] for f in range(3)], 1)
        lam, good = _lam(J + _spring_jac(q[s] - tip[s], kt, dt), dFz[s, None] * J[:, 2], ok[s])
        u = torch.zeros_like(lam)
        u[:, 2] = torch.where(good, dFz[s], torch.zeros_like(dFz[s]))
        a, p = torch.autograd.grad((fe[:, :3] * (u - lam)).sum(), (A, P))
        gA += a
        gP += p
    gP[:, 2:] = 0  # K and the pad column are not parameters of the path
    return dict(fes=fes, loss=loss, df=df, grad_atoms=gA, grad_prm=gP)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        atoms, prm = _system(case, seed)
        o, n, _ = _box(case)
        return _field(F64, atoms, prm, *_sites(case), *_axes(o, n, F64))
    if kind == "df":
        return _df_amp(_volume(case, seed), STEP, (case["tilt"], 0.5 * case["tilt"], 1.0), case["amp"])
    if kind in ("forward", "fit"):
        return None  # minutes in 64 bits; the single-molecule kinds cover the stages
    if case["npx"] * case.get("npy", case["npx"]) * case["nz"] > 2000000:
        return None
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "direct":
        return _exact_direct(case, seed)
    k, d0, Qs, QZs = synthetic.probe_params()
    if kind == "scan":
        atoms, prm, o, n, z_top = _scan_grid(case, seed)
        grid = _field(F32, atoms, prm, Qs, QZs, *_axes(o, n, F32)).to(F64)
        tip = torch.as_tensor(_raster(case["npx"], case["npy"], z_top)[:, :3], device="cuda").to(F64)
        st = _fire(lambda q, rows: _sample(grid, o, n, q)[0], tip, case["nz"], -STEP, k, d0, 1000, 1e-10, False)[::-1]
        disp = torch.stack([torch.cat([s[1] - s[3], torch.zeros_like(s[1][:, :1])], 1) for s in st], 1)
        return torch.stack([s[0] for s in st], 1), disp
    atoms, prm = _system(case, seed)
    o, n, z_end = _image_box(case)
    x = _image_raster(case)
    pts = np.zeros((len(x) ** 2, 4), np.float32)
    pts[:, 0], pts[:, 1], pts[:, 2] = np.repeat(x, len(x)), np.tile(x, len(x)), z_end + STEP * (case["nz"] - 1)
    _, st = _strokes64(case, atoms, prm, o, n, pts, z_end - 1, float(pts[0, 2]) + 1, k, d0, case["nz"], True, False, Qs,
                       QZs)
    st = st[::-1]
    fes = torch.stack([s[0] for s in st], 1).view(len(x), len(x), case["nz"], 4)
    disp = torch.stack([s[1] - s[3] for s in st], 1).view(len(x), len(x), case["nz"], 3)
    return dict(fes=fes, disp=dict(dx=disp[..., 0], dy=disp[..., 1], dz=disp[..., 2]),
                df=_df_amp(fes, STEP, (0., 0., 1.), 1.0))
