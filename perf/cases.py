"""Measured workloads of the cone-beam library.

Each case is one call (or one short solve) that a reconstruction program makes
through the package's public entry points: single projections of the operators,
the ordered-subset step, FDK on device and host arrays, whole solves and a
batch of scans.  `listed` holds fixed cases, `draw` makes further ones of the
same ranges, `prepare` builds what a program has in hand before the call (plan,
inputs on the device), `run` makes the call, `work` counts what it cannot do
without and `exact` evaluates the same result in 64 bits with plain torch.

A case is a dict: kind, volume size nx ny nz (voxels of `voxel` mm), detector W
x H of `pitch` mm, P views over `span` degrees, detector offset `offset` mm
(half-fan when not 0) and what the kind needs besides.  Source distances are
1000 / 1500 mm, 1.5 samples per voxel of nx along a ray.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

SAD, SDD, SPP = 1000.0, 1500.0, 1.5
I0 = 1.0e5          # photons per pixel of the synthetic measurements


def package():
    """The package, imported by path (its folder's name has a hyphen)."""
    name = "gt_tomography_b200"
    if name not in sys.modules:
        where = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gt-tomography_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


# ------------------------------------------------------------------ the cases
def listed():
    def c(name, kind, n, det, P, pitch, voxel=1.0, offset=0.0, span=360.0, **more):
        return dict(name=name, kind=kind, nx=n[0], ny=n[1], nz=n[2], W=det[0], H=det[1], P=P, pitch=pitch,
                    voxel=voxel, offset=offset, span=span, **more)

    return [
        # One digitally reconstructed radiograph: what an interactive preview or a 2D/3D registration calls over and over.
        c("drr_1view_128", "forward", (128, 128, 128), (256, 192), 1, 1.5, span=90.0, dtype="f32"),
        # mult_M of a whole small scan: one pixel per voxel at the isocentre, a detector twice the volume.
        c("forward_128_180v", "forward", (128, 128, 128), (256, 192), 180, 1.5, dtype="f32"),
        # The residual of one ordered-subset step of the half-fan scan of the benchmark, with its offset weight and norm.
        c("residual_256_36v", "residual", (256, 256, 256), (512, 384), 36, 0.8, offset=80.0),
        # The largest forward projection: a 512^3 volume kept in 16 bits, as a memory-bound program stores it.
        c("forward_512_bf16_12v", "forward", (512, 512, 512), (1024, 768), 12, 0.4, voxel=0.5, dtype="bf16"),
        # Odd volume and detector sizes, as a cropped region of interest has them.
        c("forward_ragged_40v", "forward", (150, 141, 93), (301, 211), 40, 0.93, dtype="f32"),
        # mult_MH of one subset into the running volume, offset-weighted.
        c("backproject_256_36v", "backproject", (256, 256, 256), (512, 384), 36, 0.8, offset=80.0, accumulate=True),
        # mult_MH of odd sizes.
        c("backproject_ragged_40v", "backproject", (150, 141, 93), (301, 211), 40, 0.93, accumulate=False),
        # FDK of the whole half-fan scan: a first image on the device.
        c("fdk_256_360v", "fdk", (256, 256, 256), (512, 384), 360, 0.8, offset=80.0, dtype="f32"),
        # FDK of a small scan on page-locked host arrays, views streamed through the device.
        c("host_fdk_128_180v", "host_fdk", (128, 128, 128), (256, 192), 180, 1.5),
        # The smallest ordered-subset step: launches and latency.
        c("step_64_8v", "step", (64, 64, 64), (128, 96), 8, 1.5, subsets=5),
        # A whole OS-MOM solve of a mid-sized scan: preconditioner, subset steps, non-negativity.
        c("osmom_160_200v", "osmom", (160, 144, 112), (320, 240), 200, 0.9, subsets=8, iterations=2),
        # Several small uneven scans solved as one batch.
        c("batch_6scans_64", "batch", (64, 64, 64), (128, 96), 60, 1.35, subsets=4, iterations=2, scans=6),
    ]


def draw(rng):
    """One more case: any kind, sizes log-uniform over the range of the listed ones, half of them odd."""
    kind = rng.choice(["forward", "forward", "residual", "backproject", "backproject", "fdk", "host_fdk", "step",
                       "osmom", "sart", "tv", "batch"])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    solve = kind in ("osmom", "sart", "tv", "batch")
    ragged = rng.random() < 0.5
    step = 1 if ragged else 8
    size = log(48, 96 if kind == "batch" else 160 if solve else 320)
    nx, ny, nz = (max(40, int(size * rng.uniform(0.8, 1.1)) // step * step) for _ in range(3))
    W = max(64, int(max(nx, ny) * rng.uniform(1.2, 2.4)) // step * step)
    H = max(48, int(W * rng.uniform(0.6, 0.8)) // step * step)
    voxel = round(rng.uniform(0.5, 1.5), 3)
    pitch = round(rng.uniform(1.05, 1.9) * 1.5 * max(nx, ny) * voxel / W, 4)
    cost = 1.2e9 if solve else 4.0e9          # ray samples per application of the operator
    most = max(1, int(cost / (W * H * SPP * nx)))
    few = 24 if solve or "fdk" in kind else 1
    P = min(log(few, 400), max(few, most))
    if kind == "host_fdk":
        P = min(P, 200)
    half_fan = kind in ("residual", "backproject", "fdk", "step", "osmom") and rng.random() < 0.4
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, W=W, H=H, P=P, pitch=pitch, voxel=voxel, span=360.0,
             offset=round(0.18 * W * pitch, 2) if half_fan else 0.0)
    if kind == "forward":
        c["dtype"] = rng.choice(["f32", "f32", "bf16", "f16"])
    if kind == "fdk":
        c["dtype"] = rng.choice(["f32", "f32", "bf16"])
    if kind == "backproject":
        c["accumulate"] = rng.random() < 0.5
    if kind == "step":
        c["subsets"] = rng.choice([4, 8, 10])
    if solve:
        c["subsets"] = rng.choice([3, 4, 8])
        c["iterations"] = rng.choice([1, 2])
    if kind == "batch":
        c["scans"] = rng.choice([3, 4, 6])
    return c


# ------------------------------------------------------------------ geometry and inputs
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def scans_of(case):
    """The scans of a batch: the case's sizes scaled by 1 to 1.5, multiples of 8; any other case is one scan."""
    if case["kind"] != "batch":
        return [case]
    out = []
    for i in range(case["scans"]):
        f = 1.0 + 0.5 * i / max(1, case["scans"] - 1)
        c = dict(case, P=int(case["P"] * (1.0 + 0.1 * i)), pitch=case["pitch"])
        for k in ("nx", "ny", "nz", "W", "H"):
            c[k] = int(case[k] * f) // 8 * 8
        c["pitch"] = case["pitch"] * case["W"] / c["W"] * f
        out.append(c)
    return out


def angles_of(case, seed):
    """Gantry angles: equal steps with the small irregularity that a real gantry has (float32, as an acquisition stores them)."""
    rng = np.random.Generator(np.random.PCG64(seed * 7919 + case["P"]))
    step = case["span"] / case["P"]
    a = (np.arange(case["P"]) + rng.uniform(-0.1, 0.1, case["P"])) * step
    a += 33.0 if case["P"] == 1 else 0.0
    return (a - a.min() if case["P"] > 1 else a).astype(np.float32)


def subset_order(case):
    """Views dealt round-robin to the subsets, subset after subset (CBSubsetOperator's order)."""
    S = case["subsets"]
    return np.concatenate([np.arange(s, case["P"], S) for s in range(S)]).astype(np.int64)


def ellipsoids(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    L = np.array([case["nx"], case["ny"], case["nz"]]) * case["voxel"]
    e = np.zeros((8, 7))
    e[:, 0:3] = rng.uniform(-0.25, 0.25, (8, 3)) * L
    e[:, 3:6] = rng.uniform(0.05, 0.3, (8, 3)) * L
    e[:, 6] = rng.uniform(0.002, 0.02, 8)
    e[0, :6] = [0, 0, 0, *(0.42 * L)]
    return e


def volume(case, seed):
    """Attenuation values (1/mm): a body of ellipsoids with a little texture."""
    dev = device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    v = 0.0005 * torch.rand((case["nz"], case["ny"], case["nx"]), generator=gen, device=dev)
    axes = [(torch.arange(n, device=dev, dtype=torch.float32) + 0.5 - n / 2) * case["voxel"]
            for n in (case["nz"], case["ny"], case["nx"])]
    for cx, cy, cz, ax, ay, az, rho in ellipsoids(case, seed):
        q = (((axes[0] - cz) / az) ** 2)[:, None, None] + (((axes[1] - cy) / ay) ** 2)[None, :, None] \
            + (((axes[2] - cx) / ax) ** 2)[None, None, :]
        v += rho * (q < 1.0)
    return v.contiguous()


def measured(case, seed, angles):
    """Line integrals through the ellipsoids with Poisson noise, (P, H, W) float32 in the order of `angles`."""
    dev = device()
    e = ellipsoids(case, seed)
    W, H = case["W"], case["H"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed + 1)
    out = torch.empty((len(angles), H, W), dtype=torch.float32, device=dev)
    u = ((torch.arange(W, device=dev, dtype=torch.float32) + 0.5) / W - 0.5) * W * case["pitch"] + case["offset"]
    v = ((torch.arange(H, device=dev, dtype=torch.float32) + 0.5) / H - 0.5) * H * case["pitch"]
    for p0 in range(0, len(angles), 32):
        th = torch.from_numpy(angles[p0:p0 + 32]).to(dev) * (math.pi / 180.0)
        c, s = torch.cos(th)[:, None, None], torch.sin(th)[:, None, None]
        dx, dy = c * u - s * SDD, s * u + c * SDD     # detector point minus source, (views, 1, W)
        dx, dy = dx.reshape(-1, 1, W), dy.reshape(-1, 1, W)
        dz = v[None, :, None]
        length = torch.sqrt(dx * dx + dy * dy + dz * dz)
        line = torch.zeros((th.numel(), H, W), dtype=torch.float32, device=dev)
        for cx, cy, cz, ax, ay, az, rho in e:
            ox, oy, oz = (SAD * s - cx) / ax, (-SAD * c - cy) / ay, -cz / az
            qa = (dx / ax) ** 2 + (dy / ay) ** 2 + (dz / az) ** 2
            qb = ox * dx / ax + oy * dy / ay + oz * dz / az
            qc = ox * ox + oy * oy + oz * oz - 1.0
            line += rho * 2.0 * torch.sqrt(torch.clamp(qb * qb - qa * qc, min=0.0)) / qa * length
        counts = torch.poisson(I0 * torch.exp(-line), generator=gen)
        out[p0:p0 + 32] = -torch.log(torch.clamp(counts, min=1.0) / I0)
    return out


def hann_ramp(W):
    k = np.arange(W + 1, dtype=np.float64)
    h = k * 0.5 * (1.0 + np.cos(np.pi * k / W))
    return (h * ((W + 1) / np.abs(h).sum())).astype(np.float32)


def preconditioner(case, seed):
    """Positive per-voxel steps of the size that 1 / (A^T A 1) has."""
    gen = torch.Generator(device=device())
    gen.manual_seed(seed + 2)
    full = case["P"] * case["subsets"] * max(case["nx"], case["ny"]) * case["voxel"]
    shape = (case["nz"], case["ny"], case["nx"])
    return ((0.8 + 0.4 * torch.rand(shape, generator=gen, device=device())) / full).contiguous()


def geometry(case):
    L = package()._lib
    m = case["voxel"]
    return L.CbctGeometry(SAD, SDD, case["W"] * case["pitch"], case["H"] * case["pitch"], case["W"], case["H"],
                          case["nx"], case["ny"], case["nz"], case["nx"] * m, case["ny"] * m, case["nz"] * m, SPP)


def offsets_of(case, n):
    return np.tile(np.array([[case["offset"], 0.0]], np.float32), (n, 1))


def acquisition(case, angles, projections):
    gtb = package()
    geo = gtb.CBCT_geometry(SAD, SDD, (case["W"] * case["pitch"], case["H"] * case["pitch"]), angles.copy(),
                            offsets_of(case, len(angles)))
    return gtb.CBCT_acquisition(geo, projections)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    gtb = package()
    kind = case["kind"]
    dev = device()
    angles = angles_of(case, seed)
    P = case["P"]
    off = int(case["offset"] != 0.0)
    st = dict(kind=kind, case=case)
    if kind in ("forward", "residual", "backproject", "fdk"):
        st["plan"] = gtb.Plan(geometry(case), angles, offsets_of(case, P), None, [off])
    if kind == "forward":
        st["vol"] = volume(case, seed).to(DTYPES[case["dtype"]]).contiguous()
        st["code"] = {"f32": gtb.CBCT_F32, "bf16": gtb.CBCT_BF16, "f16": gtb.CBCT_F16}[case["dtype"]]
        st["out"] = torch.empty(st["plan"].proj_shape(), dtype=torch.float32, device=dev)
    elif kind == "residual":
        st["vol"] = volume(case, seed)
        st["b"] = measured(case, seed + 100, angles)
        st["out"] = torch.empty_like(st["b"])
        st["norm2"] = torch.zeros(1, dtype=torch.float64, device=dev)
    elif kind == "backproject":
        st["proj"] = measured(case, seed, angles)
        st["out"] = torch.zeros(st["plan"].vol_shape, dtype=torch.float32, device=dev)
    elif kind == "fdk":
        st["proj"] = measured(case, seed, angles).to(DTYPES[case["dtype"]]).contiguous()
        st["filter"] = hann_ramp(case["W"])
        st["flags"] = gtb._lib.CBCT_FDK_OFFSET if off else 0
        st["out"] = torch.empty(st["plan"].vol_shape, dtype=torch.float32, device=dev)
    elif kind == "host_fdk":
        host = measured(case, seed, angles).cpu()
        E = gtb.hoCuConebeamProjectionOperator()
        E.setup(acquisition(case, angles, host.numpy()), None,
                (case["nx"] * case["voxel"], case["ny"] * case["voxel"], case["nz"] * case["voxel"]),
                is_dims=(case["nx"], case["ny"], case["nz"]))
        E.set_use_filtered_backprojection(True)
        E.set_frequency_filter(hann_ramp(case["W"]))
        st["E"], st["proj"] = E, host.pin_memory()
        st["out"] = torch.zeros((case["nz"], case["ny"], case["nx"]), dtype=torch.float32).pin_memory()
    elif kind == "step":
        st["plan"] = gtb.Plan(geometry(case), angles, offsets_of(case, P), None, [off])
        st["z"] = volume(case, seed)
        st["xold"] = (0.9 * st["z"]).contiguous()
        st["precon"] = preconditioner(case, seed)
        st["b"] = measured(case, seed + 100, angles)
        st["r"] = torch.empty_like(st["b"])
        st["norm2"] = torch.zeros(1, dtype=torch.float64, device=dev)
    elif kind in ("osmom", "sart", "tv"):
        proj = measured(case, seed, angles).cpu().numpy()
        acq = acquisition(case, angles, proj)
        E = gtb.CBSubsetOperator(case["subsets"])
        E.set_use_offset_correction(bool(off))
        E.setup(acq, None, (case["nx"] * case["voxel"], case["ny"] * case["voxel"], case["nz"] * case["voxel"]),
                is_dims=(case["nx"], case["ny"], case["nz"]))
        solver = gtb.osSARTSolver() if kind == "sart" else gtb.osMOMSolverD()
        solver.set_max_iterations(case["iterations"])
        solver.set_non_negativity_constraint(True)
        solver.set_encoding_operator(E)
        if kind == "tv":
            tv = gtb.cuTVPrimalDualOperator(0.02)
            tv.set_weight(0.5)
            solver.add_regularization_operator(tv)
            solver.set_reg_steps(2)
        st["solver"], st["b"] = solver, torch.from_numpy(acq.projections).to(dev)
    elif kind == "batch":
        jobs = []
        for i, sc in enumerate(scans_of(case)):
            order = subset_order(sc)
            a = angles_of(sc, seed + i)[order]
            sizes = [len(range(s, sc["P"], sc["subsets"])) for s in range(sc["subsets"])]
            plan = gtb.Plan(geometry(sc), a, offsets_of(sc, sc["P"]), sizes, [0] * sc["subsets"])
            jobs.append(dict(plan=plan, b=measured(sc, seed + i, a), iterations=sc["iterations"], nonneg=True,
                             z=torch.empty(plan.vol_shape, dtype=torch.float32, device=dev)))
        st["jobs"] = jobs
    return st


def run(state):
    gtb = package()
    kind = state["kind"]
    if kind == "forward":
        return state["plan"].forward(state["vol"], state["out"], -1, False, state["code"])
    if kind == "residual":
        state["plan"].forward_residual(state["vol"], state["b"], state["out"], -1, 1.0,
                                       state["case"]["offset"] != 0.0, state["norm2"])
        return state["out"], state["norm2"]
    if kind == "backproject":
        return state["plan"].backproject(state["proj"], state["out"], -1, 0, True, state["case"]["accumulate"])
    if kind == "fdk":
        return state["plan"].fdk(state["proj"], state["out"], state["filter"], state["flags"])
    if kind == "host_fdk":
        return state["E"].mult_MH(state["proj"], state["out"])
    if kind == "step":
        state["plan"].osmom_step(0, state["b"], state["z"], state["xold"], state["precon"], state["r"],
                                 float(state["case"]["subsets"]), 0.25, True, state["norm2"])
        return state["z"], state["xold"], state["r"], state["norm2"]
    if kind in ("osmom", "sart", "tv"):
        return state["solver"].solve(state["b"])
    gtb.batch_osmom(state["jobs"], fused=True)
    return [j["z"] for j in state["jobs"]]


# ------------------------------------------------------------------ work
def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    for sc in scans_of(case):
        vox = float(sc["nx"]) * sc["ny"] * sc["nz"]
        pix = float(sc["W"]) * sc["H"] * sc["P"]
        columns = float(sc["W"]) * sc["P"]
        N = int(SPP * sc["nx"])
        # Forward: in-plane interpolation of every column sample on every plane (3 lerps of 3 flops), then per ray
        # sample its lerp along z and the sum.  Back-projection: a bilinear tap and the sum per voxel and view.
        fwd, bwd = columns * N * (9.0 * min(sc["nz"], sc["H"])) + pix * N * 4.0, vox * sc["P"] * 10.0
        vs = 2.0 if sc.get("dtype") in ("bf16", "f16") else 4.0
        kind = sc["kind"]
        if kind == "forward":
            b, f = vs * vox + 4 * pix, fwd
        elif kind == "residual":
            b, f = 4 * vox + 8 * pix, fwd
        elif kind == "backproject":
            b, f = 4 * pix + (8 if sc["accumulate"] else 4) * vox, bwd
        elif kind in ("fdk", "host_fdk"):
            length = 2 ** math.ceil(math.log2(2 * sc["W"]))
            b, f = vs * pix + 4 * vox, bwd + sc["H"] * sc["P"] * 5.0 * length * math.log2(length)
        elif kind == "step":
            b, f = 4 * (5 * vox) + 8 * pix, fwd + bwd
        else:
            passes = sc["iterations"] + (1.0 if kind != "sart" else 2.0)
            b, f = 4 * (vox + pix), passes * (fwd + bwd)
        total["bytes"] += b
        total["flops"] += f
    return total


# ------------------------------------------------------------------ exact (64 bits, plain torch)
F64 = torch.float64


def e_forward(case, vol, angles):
    """Ray sums of mult_M: N equidistant trilinear samples between the clips of the ray, times their spacing."""
    dev = vol.device
    n = [case["nx"], case["ny"], case["nz"]]
    Lmm = [float(np.float32(k * case["voxel"])) for k in n]
    W, H, N = case["W"], case["H"], int(np.float32(SPP) * np.float32(case["nx"]))
    fu, fv = float(np.float32(W * case["pitch"])), float(np.float32(H * case["pitch"]))
    off = float(np.float32(case["offset"]))
    q = ((torch.arange(W, device=dev, dtype=F64) + 0.5) / W - 0.5) * fu + off
    r = ((torch.arange(H, device=dev, dtype=F64) + 0.5) / H - 0.5) * fv
    out = torch.empty((len(angles), H, W), dtype=F64, device=dev)
    k = torch.arange(N, device=dev, dtype=F64)
    rows = max(1, int(2.0e7 / (W * N)))
    grid_in = vol[None, None].to(F64)
    for p, a in enumerate(angles):
        th = float(a) * math.pi / 180.0
        c, s = math.cos(th), math.sin(th)
        S = [SAD * s, -SAD * c, 0.0]
        for v0 in range(0, H, rows):
            rr = r[v0:v0 + rows]
            d = [(c * q - s * (SDD - SAD) - S[0]).expand(len(rr), W), (s * q + c * (SDD - SAD) - S[1]).expand(len(rr), W),
                 rr[:, None].expand(len(rr), W)]
            lo = hi = None
            for i in range(3):
                t1, t2 = (Lmm[i] / 2 - S[i]) / d[i], (-Lmm[i] / 2 - S[i]) / d[i]
                mn, mx = torch.minimum(t1, t2), torch.maximum(t1, t2)
                lo = mn if lo is None else torch.maximum(lo, mn)
                hi = mx if hi is None else torch.minimum(hi, mx)
            a1, a2 = torch.clamp(lo, min=0.0), torch.clamp(hi, max=1.0)
            length = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            delta = (a2 - a1).abs() * length / N
            t = a1[..., None] + ((a2 - a1) / N)[..., None] * k
            axes = []
            for i in range(3):
                texel = ((S[i] + t * d[i][..., None]) / Lmm[i] + 0.5) * n[i] - 0.5
                axes.append(2.0 * texel / (n[i] - 1) - 1.0)
            g = torch.stack(axes, -1)[None]
            val = torch.nn.functional.grid_sample(grid_in, g, mode="bilinear", padding_mode="zeros", align_corners=True)
            out[p, v0:v0 + rows] = val[0, 0].sum(-1) * delta
    return out


def e_offset(case, proj):
    """The sin^2 half-fan weight of mult_MH."""
    o = float(np.float32(case["offset"]))
    if o == 0.0:
        return proj
    W, fu = case["W"], float(np.float32(case["W"] * case["pitch"]))
    omega = fu / 2 - abs(o)
    t = (fu * (torch.arange(W, device=proj.device, dtype=F64) / W - 0.5) + o) * math.copysign(1.0, o)
    w = torch.where(t.abs() <= omega, torch.sin(math.pi * (t + omega) / (4 * omega)) ** 2, torch.ones_like(t))
    return proj * torch.where(t < -omega, torch.zeros_like(w), w)


def e_backproject(case, proj, angles, fdk=False):
    dev = proj.device
    n = [case["nx"], case["ny"], case["nz"]]
    Lmm = [float(np.float32(k * case["voxel"])) for k in n]
    W, H = case["W"], case["H"]
    fu, fv = float(np.float32(W * case["pitch"])), float(np.float32(H * case["pitch"]))
    off = float(np.float32(case["offset"]))
    x, y, z = (((torch.arange(m, device=dev, dtype=F64) + 0.5) / m - 0.5) * l for m, l in zip(n, Lmm))
    out = torch.zeros((n[2], n[1], n[0]), dtype=F64, device=dev)
    for p, a in enumerate(angles):
        th = float(a) * math.pi / 180.0
        c, s = math.cos(th), math.sin(th)
        xr, yr = c * x[None, :] + s * y[:, None], -s * x[None, :] + c * y[:, None]
        cu = ((SDD * xr / (yr + SAD) - off) / fu + 0.5) * W - 0.5
        gu = (2.0 * cu / (W - 1) - 1.0)[None].expand(n[2], n[1], n[0])
        cv = ((SDD * z[:, None, None] / (yr + SAD)) / fv + 0.5) * H - 0.5
        g = torch.stack([gu, 2.0 * cv / (H - 1) - 1.0], -1).reshape(1, n[2] * n[1], n[0], 2)
        val = torch.nn.functional.grid_sample(proj[p][None, None], g, mode="bilinear", padding_mode="zeros",
                                              align_corners=True).reshape(n[2], n[1], n[0])
        out += val / (1.0 - yr / SAD) ** 2 if fdk else val
    return out


def e_fdk(case, proj, angles):
    W, H = case["W"], case["H"]
    dev = proj.device
    fu, fv = float(np.float32(W * case["pitch"])), float(np.float32(H * case["pitch"]))
    s = SAD * (torch.arange(W, device=dev, dtype=F64) / W - 0.5) * fu / SDD
    v = SAD * (torch.arange(H, device=dev, dtype=F64) / H - 0.5) * fv / SDD
    p = proj * (SAD / torch.sqrt(SAD * SAD + s[None, :] ** 2 + v[:, None] ** 2)).float().double()
    filt = torch.from_numpy(hann_ramp(W)).to(dev).double()
    for i in range(0, p.shape[0], 32):
        row = torch.fft.irfft(torch.fft.rfft(p[i:i + 32], n=2 * W, dim=-1) * filt, n=2 * W, dim=-1)
        p[i:i + 32] = row[..., :W]
    return e_backproject(case, e_offset(case, p), angles, True) * (2.0 / len(angles))


def e_subsets(case):
    S, P = case["subsets"], case["P"]
    sizes = [len(range(s, P, S)) for s in range(S)]
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    return [slice(int(f), int(f + n)) for f, n in zip(first, sizes)]


def e_tv(x, s, D, lam, alpha, tau, steps, gam):
    sigma = 1.0 / (tau * 16.0)
    for _ in range(steps):
        scale = sigma / (1.0 + sigma * alpha)
        d = [(torch.roll(x, -1, dims) - x) * scale for dims in (2, 1, 0)]
        m = torch.clamp(torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2), min=1.0)
        d = [q / m for q in d]
        gv = sum(torch.roll(q, 1, dims) - q for q, dims in zip(d, (2, 1, 0)))
        x = ((x - tau * gv) + tau / lam * (s / D)) / ((1.0 / D) * (tau / lam) + 1.0)
        theta = 1.0 / math.sqrt(1.0 + 2.0 * gam * tau)
        tau, sigma = tau * theta, sigma / theta
    return x


def e_osmom(case, b, angles, tv=None):
    subsets = e_subsets(case)
    S = len(subsets)
    ones = torch.ones((case["nz"], case["ny"], case["nx"]), dtype=F64, device=b.device)
    pre = sum(e_backproject(case, e_offset(case, e_forward(case, ones, angles[s])), angles[s]) for s in subsets)
    D = 1.0 / torch.clamp(pre, min=1e-6)
    gam = 0.35 / tv["weight"] / (D.numel() / float(D.abs().sum())) if tv else 0.0
    z = torch.zeros_like(ones)
    xold = z.clone()
    t = told = 1.0
    for _ in range(case["iterations"]):
        for s in subsets:
            t = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
            g = e_backproject(case, e_offset(case, e_forward(case, z, angles[s]) - b[s]), angles[s])
            step = z - S * (D * g)
            x = e_tv(z, step, D, tv["weight"], tv["alpha"], 1e-3, tv["steps"], gam) if tv else step
            x = torch.clamp(x, min=0.0)
            m = (told - 1.0) / t
            z = x * (1.0 + m) - m * xold
            xold, told = x, t
    return z


def e_sart(case, b, angles):
    subsets = e_subsets(case)
    ones = torch.ones((case["nz"], case["ny"], case["nx"]), dtype=F64, device=b.device)
    Wp = 1.0 / torch.clamp(e_forward(case, ones, angles), min=1e-6)
    V = [1.0 / torch.clamp(e_backproject(case, e_offset(case, torch.ones_like(b[s])), angles[s]), min=1e-6)
         for s in subsets]
    x = torch.zeros_like(ones)
    order = list(range(len(subsets)))
    for _ in range(case["iterations"]):
        for i in order:
            s = subsets[i]
            r = -(e_forward(case, x, angles[s]) - b[s]) * Wp[s]
            x = torch.clamp(x + V[i] * e_backproject(case, e_offset(case, r), angles[s]), min=0.0)
        order.reverse()
    return x


def exact(case, seed):
    samples = float(case["W"]) * case["H"] * case["P"] * SPP * case["nx"]
    passes = case.get("iterations", 0) + 1
    if not torch.cuda.is_available() and samples * passes > 2e7:
        return None
    kind = case["kind"]
    angles = angles_of(case, seed)
    if kind == "forward":
        return e_forward(case, volume(case, seed).to(DTYPES[case["dtype"]]), angles)
    if kind == "residual":
        d = e_forward(case, volume(case, seed), angles) - measured(case, seed + 100, angles).double()
        return e_offset(case, d), (d * d).sum().reshape(1)
    if kind == "backproject":
        # an accumulating call adds to what its earlier passes left: the first pass starts from zeros
        return e_backproject(case, e_offset(case, measured(case, seed, angles).double()), angles)
    if kind == "fdk":
        return e_fdk(case, measured(case, seed, angles).to(DTYPES[case["dtype"]]).double(), angles)
    if kind == "host_fdk":
        return e_fdk(case, measured(case, seed, angles).double(), angles - angles.min()).cpu()
    if kind == "step":
        z = volume(case, seed)
        xold = (0.9 * z).double()
        z = z.double()
        d = e_forward(case, z, angles) - measured(case, seed + 100, angles).double()
        r = e_offset(case, d)
        zt = z - case["subsets"] * (preconditioner(case, seed).double() * e_backproject(case, r, angles))
        x = torch.clamp(zt, min=0.0)
        return x * 1.25 - 0.25 * xold, x, r, (d * d).sum().reshape(1)
    if kind in ("osmom", "sart", "tv"):
        order = subset_order(case)
        # the measurement is made in acquisition order and permuted, as setup does
        b = measured(case, seed, angles)[torch.from_numpy(order).to(device())].double()
        a = (angles - angles.min())[order]
        if kind == "sart":
            return e_sart(case, b, a)
        return e_osmom(case, b, a, dict(weight=0.5, alpha=0.02, steps=2) if kind == "tv" else None)
    out = []
    for i, sc in enumerate(scans_of(case)):
        a = angles_of(sc, seed + i)[subset_order(sc)]
        out.append(e_osmom(sc, measured(sc, seed + i, a).double(), a))
    return out
