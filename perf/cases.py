"""Representative calls of the Fourier-slice operators, from the smallest to the largest.

Each case is one call (or one forward + backward pass) that programs built on this package make:
projecting reconstructions, back-projecting slices into them, and the gradients of both.  The
boxes, pose counts and options are those of the benchmark's configurations and of the tests, or
plain sizes of the same kind; ``draw`` gives more of the same ranges.  Everything is synthetic:
volumes are spectra of noise that falls off with frequency, slices are complex noise with
CTF^2-like weights in [0, 1], poses are uniform rotations with shifts of a few pixels.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("torch-projectors_b200"))
import torch_projectors_b200 as tp  # noqa: E402

# What a case's "op" does:
#   project      project_2d_forw / project_3d_to_2d_forw without gradients (simulating slices, scoring)
#   step         the same with gradients: out = project(...), then the gradients of the reconstruction,
#                rotations and shifts ("rec": the reconstruction is optimised too, else it is fixed)
#   backproject  backproject_2d_forw / backproject_2d_to_3d_forw without gradients (class averages, reconstructions)
#   accumulate   one chunk of a streamed 3D reconstruction into its persistent accumulator
#   backstep     back-projection with gradients of the slices, weights, rotations and shifts


def _case(name, op, dim, box, os_, poses, *, batch=1, cubic=False, weights=True, rec=True, shift=4.0, double=False, cutoff=0.0):
    """box: of the slices; os_: oversampling of the reconstruction; cutoff: share of Nyquist (0: the default)."""
    c = {"op": op, "dim": dim, "box": box, "os": os_, "poses": poses, "batch": batch, "cubic": cubic, "weights": weights, "rec": rec,
         "shift": shift, "double": double, "cutoff": cutoff}
    return dict(c, name=name) if name else c


def listed():
    return [
        # scoring one 2D reference: a few hundred rotated copies of a small image, called in a loop where the latency counts
        _case("project_2d_small", "project", 2, 64, 2.0, 256),
        # checking a model's gradients in double precision on a small volume: launches and host work count
        _case("step_3d_double", "step", 3, 32, 2.0, 50, cubic=True, double=True),
        # 2D class averages: eight classes, each with its own slices, weights and poses
        _case("backproject_2d_classes", "backproject", 2, 128, 2.0, 1000, batch=8),
        # refining eight 2D references together with the poses of their members
        _case("step_2d_classes", "step", 2, 128, 2.0, 500, batch=8, cubic=True),
        # simulating a data set from one volume: box-256 oversampled volume, 10,000 poses, cubic, explicit radius cutoff
        _case("project_3d_cubic", "project", 3, 128, 2.0, 10000, cubic=True, shift=8.0, cutoff=1.0),
        # quick linear projections at the volume's own sampling, with a box and a pose count that fill no tile
        _case("project_3d_linear", "project", 3, 180, 1.0, 3001, shift=5.0),
        # weighted reconstruction from 50,000 slices, linear
        _case("backproject_3d_linear", "backproject", 3, 128, 2.0, 50000, shift=8.0),
        # cubic reconstruction of a small data set, ragged box
        _case("backproject_3d_cubic", "backproject", 3, 90, 2.0, 2501, cubic=True),
        # one optimiser step over volume, rotations and shifts: box-512 oversampled volume, 4,096 poses, cubic
        _case("step_3d", "step", 3, 256, 2.0, 4096, cubic=True, shift=10.0),
        # pose refinement against a fixed volume, linear
        _case("step_3d_poses", "step", 3, 128, 2.0, 4096, rec=False),
        # one chunk of a streamed high-resolution reconstruction (box 400 into box 800), the largest case
        _case("accumulate_3d", "accumulate", 3, 400, 2.0, 8192, shift=12.0),
        # learning through a back-projection: gradients of slices, weights and poses
        _case("backstep_3d", "backstep", 3, 64, 2.0, 2000),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    while True:
        op = rng.choice(["project", "project", "step", "step", "backproject", "backproject", "accumulate", "backstep"])
        dim = 3 if op == "accumulate" else rng.choice([2, 3, 3])
        double = op in ("project", "step", "backproject") and rng.random() < 0.1
        box = 2 * int(log(16, 64 if double else 200))
        c = _case(None, op, dim, box, rng.choice([1.0, 1.5, 2.0, 2.0]), int(log(8, 60000)),
                  batch=rng.choice([1, 1, 1, 2, 5, 8]) if dim == 2 else rng.choice([1, 1, 1, 1, 2]),
                  cubic=rng.random() < 0.5, weights=op == "accumulate" or rng.random() < 0.75, rec=rng.random() < 0.6,
                  shift=round(rng.uniform(2.0, 12.0), 2), double=double, cutoff=rng.choice([0.0, 0.0, 0.0, 0.8, 1.0]))
        # no more work than the largest listed cases, and a state of a few GB
        if _sums(c) <= (5e8 if double else 6e9) and work(c)["bytes"] <= 6e9:
            return c


def _sizes(c):
    N = c["box"]
    raw = math.ceil(N * c["os"])
    R = raw + raw % 2
    return N, N // 2 + 1, R, R // 2 + 1


def _rotations(dim, B, P, gen, dtype):
    if dim == 2:
        a = torch.rand(B * P, generator=gen, device="cuda", dtype=torch.float64) * (2 * math.pi)
        m = torch.stack([a.cos(), -a.sin(), a.sin(), a.cos()], 1)
    else:
        q = torch.randn(B * P, 4, generator=gen, device="cuda", dtype=torch.float64)
        w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
        m = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                         2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                         2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)
    return m.reshape(B, P, dim, dim).to(dtype).contiguous()


def _spectrum(shape, gen, dtype):
    """Complex noise in rfft layout whose amplitude falls off with the distance from the origin."""
    R = shape[1]
    k = torch.fft.fftfreq(R, device="cuda").square()
    h = torch.fft.rfftfreq(R, device="cuda").square()
    r2 = k[:, None] + h if len(shape) == 3 else k[:, None, None] + k[:, None] + h
    v = torch.randn(shape, generator=gen, device="cuda", dtype=torch.complex64)
    return v.div_(1.0 + 8.0 * r2.sqrt()).to(dtype)


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    cplx, real = (torch.complex128, torch.float64) if case["double"] else (torch.complex64, torch.float32)
    N, Nh, R, Rh = _sizes(case)
    B, P, dim, op = case["batch"], case["poses"], case["dim"], case["op"]
    grads = op in ("step", "backstep")
    s = {"case": case}
    s["rot"] = _rotations(dim, B, P, gen, real).requires_grad_(grads)
    s["shifts"] = ((torch.rand(B, P, 2, generator=gen, device="cuda", dtype=real) * 2 - 1) * case["shift"]).requires_grad_(grads)
    s["kw"] = {"interpolation": "cubic" if case["cubic"] else "linear", "oversampling": case["os"]}
    if case["cutoff"]:
        s["kw"]["fourier_radius_cutoff"] = case["cutoff"] * N / 2
    rec_shape, slices = (B,) + (R,) * (dim - 1) + (Rh,), (B, P, N, Nh)
    if op in ("project", "step"):
        s["rec"] = _spectrum(rec_shape, gen, cplx).requires_grad_(op == "step" and case["rec"])
        s["kw"]["output_shape"] = (N, N)
        if op == "step":
            s["grad"] = torch.randn(slices, generator=gen, device="cuda", dtype=cplx)
    else:
        s["proj"] = torch.randn(slices, generator=gen, device="cuda", dtype=cplx).requires_grad_(grads)
        s["w"] = torch.rand(slices, generator=gen, device="cuda", dtype=real).requires_grad_(grads) if case["weights"] else None
        if op == "accumulate":
            s["acc"] = tp.new_backprojection_accumulator(B, R, "cuda")
        elif op == "backstep":
            s["grad"] = torch.randn(rec_shape, generator=gen, device="cuda", dtype=cplx)
            s["grad_w"] = torch.randn(rec_shape, generator=gen, device="cuda", dtype=real)
    return s


def run(s):
    case = s["case"]
    op, two = case["op"], case["dim"] == 2
    if op in ("project", "step"):
        project = tp.project_2d_forw if two else tp.project_3d_to_2d_forw
        out = project(s["rec"], s["rot"], s["shifts"], **s["kw"])
        if op == "project":
            return out
        wanted = ([s["rec"]] if case["rec"] else []) + [s["rot"], s["shifts"]]
        return [out.detach(), *torch.autograd.grad(out, wanted, s["grad"])]
    if op == "accumulate":
        tp.backproject_2d_to_3d_accumulate_interleaved_(s["acc"], s["proj"], s["rot"], s["w"], s["shifts"], **s["kw"])
        return s["acc"]
    backproject = tp.backproject_2d_forw if two else tp.backproject_2d_to_3d_forw
    data, weight = backproject(s["proj"], s["rot"], s["w"], s["shifts"], **s["kw"])
    if op == "backproject":
        return [data, weight] if case["weights"] else data
    outs, seeds, wanted = [data], [s["grad"]], [s["proj"], s["rot"], s["shifts"]]
    if case["weights"]:
        outs, seeds, wanted = outs + [weight], seeds + [s["grad_w"]], wanted + [s["w"]]
    return [o.detach() for o in outs] + list(torch.autograd.grad(outs, wanted, seeds))


def _pixels(c):
    """Pixels inside the cutoff, of all slices."""
    r = c["box"] / 2 * (c["cutoff"] or 1.0)
    return c["batch"] * c["poses"] * (math.pi / 2 * r * r + r)


def _sums(c):
    """Voxels that are read or added to, over all pixels of the forward pass."""
    return _pixels(c) * (4 if c["cubic"] else 2) ** c["dim"]


def work(case):
    N, Nh, R, Rh = _sizes(case)
    B, P, dim, op = case["batch"], case["poses"], case["dim"], case["op"]
    unit = 2 if case["double"] else 1
    vox, pix = B * R ** (dim - 1) * Rh, B * P * N * Nh
    inside = min(_pixels(case), pix)
    poses = B * P * (dim * dim + 2) * 4 * unit
    w = 4 * unit if case["weights"] else 0
    c8 = 8 * unit
    taps = _sums(case)
    if op == "project":
        return {"bytes": vox * c8 + pix * c8 + poses, "flops": 4 * taps}
    if op == "step":            # out; its gradient in; the reconstruction's gradient out; the poses' gradients out
        return {"bytes": vox * c8 * (2 if case["rec"] else 1) + pix * c8 + inside * c8 + 2 * poses,
                "flops": (4 + 4 * dim + (4 if case["rec"] else 0)) * taps}
    if op == "backproject":     # the pixels inside the cutoff in, the volumes out
        return {"bytes": inside * (c8 + w) + vox * (c8 + w) + poses, "flops": (6 if w else 4) * taps}
    if op == "accumulate":      # the accumulator is read and written
        return {"bytes": inside * 12 + 2 * vox * 16 + poses, "flops": 6 * taps}
    return {"bytes": inside * (c8 + w) + pix * (c8 + w) + 2 * vox * (c8 + w) + 2 * poses, "flops": (4 + 4 + 4 * dim + (4 if w else 0)) * taps}


def tolerance(case):
    # single precision: sums of up to a few thousand terms in an order that is not fixed; double: the same at 2^-53
    return {"rel": 1e-12} if case["double"] else {"rel": 1e-5}
