"""The cell-sorted scatters (pixels listed by brick, sums per cell in registers) against the CPU oracle, at sizes and poses where the
lists can go wrong: one brick and several, ragged boxes, boxes that are not N times the oversampling, several passes over
the list, batches, cutoffs inside and beyond Nyquist, samples on the lattice and out of the grid, values that are not finite."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from cases import Case, TOL_ATOMIC, axis_aligned_rotations, make_inputs, rel_err

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

#      B  P   N   R   os    cutoff  B_rot  B_shift
SIZES = [(1, 40, 4, 8, 2.0, None, 1, 1),
         (1, 45, 18, 36, 2.0, None, 1, 1),
         (2, 33, 20, 30, 1.5, 7.3, 2, 0),
         (2, 9, 34, 34, 1.0, 20.0, 1, 2),           # cutoff beyond Nyquist: corners of the slices, out of the grid
         (1, 37, 26, 34, 1.25, None, 1, 1),
         (3, 7, 30, 40, 2.0, 14.2, 1, 1),           # the box is smaller than N times the oversampling
         (1, 3, 48, 120, 2.0, 17.0, 1, 1),
         (1, 700, 18, 36, 2.0, None, 1, 1)]         # several batches in a brick
LARGE = [(1, 30, 20, 340, 17.0, None, 1, 1)]        # 44,528 bricks: one counter of each in global memory
SIZES_2D = SIZES + [(2, 300, 70, 140, 2.0, 33.0, 2, 2), (1, 23, 400, 640, 1.5, None, 1, 1)]


def _inputs(dim, interp, size, seed):
    B, P, N, R, os_, cutoff, B_rot, B_shift = size
    t = make_inputs(Case("lists", dim, interp, B, P, N, R, os_, cutoff, B_rot, B_shift, shift_range=5.0, seed=seed))
    lattice = axis_aligned_rotations(torch.Generator().manual_seed(seed)) if dim == 3 else t["rot"][0, :0]
    if P >= len(lattice) + 4:
        t["rot"][0, 2: 2 + len(lattice)] = lattice
        t["rot"][0, -1] *= 1.3                          # magnified, sheared, singular
        t["rot"][0, -2, :, 1] += 0.7 * t["rot"][0, -2, :, 0]
        t["rot"][0, -3, :, 1] = t["rot"][0, -3, :, 0]
    return t


def check():
    """In a fresh process with the lists forced on (the library reads the switches once)."""
    sys.path[:0] = [str(ROOT), str(ROOT / "torch-projectors_b200"), str(ROOT / "tests")]
    import torch_projectors_b200 as tp
    from oracle import port
    lib = tp._abi.load()
    for dim in (3, 2):
        gradient, back = (tp.project_3d_to_2d_forw, port.project_3d_to_2d_back) if dim == 3 else (tp.project_2d_forw, port.project_2d_back)
        forw, ref = (tp.backproject_2d_to_3d_forw, port.backproject_2d_to_3d_forw) if dim == 3 else (tp.backproject_2d_forw, port.backproject_2d_forw)
        for seed, size in enumerate((SIZES if dim == 3 else SIZES_2D) + (LARGE if os.environ.get("B200PROJ_LIST_SHARED") == "4096" else [])):
            B, P, N, R, os_, cutoff = size[:6]
            for interp in ("linear", "cubic"):
                t = _inputs(dim, interp, size, seed)
                c = {k: v.cuda() if v is not None else None for k, v in t.items()}
                radius = N / 2.0 if cutoff is None else cutoff
                code = tp.ops._interp_code(interp)
                assert lib.b200proj_scatter_workspace_bytes(dim, B, P, N, code, 1, os_, radius) > 0 and lib.b200proj_gradient_workspace_bytes(dim, B, R, P, N, code, 0, os_, radius) > 0
                rec = c["rec"].requires_grad_(True)
                out = gradient(rec, c["rot"], c["shifts"], output_shape=(N, N), interpolation=interp, oversampling=os_, fourier_radius_cutoff=cutoff)
                out.backward(c["proj"])
                want = back(t["proj"], t["rec"], t["rot"], t["shifts"], interp, os_, cutoff)[0]
                assert rel_err(rec.grad, want) <= TOL_ATOMIC, (dim, size, interp, "gradient", rel_err(rec.grad, want))
                kw = dict(interpolation=interp, oversampling=os_, fourier_radius_cutoff=cutoff)
                for weights in (None, "weights"):
                    data, wrec = forw(c["proj"], c["rot"], c[weights] if weights else None, c["shifts"], **kw)
                    d, w = ref(t["proj"], t[weights] if weights else None, t["rot"], t["shifts"], interp, os_, cutoff)
                    assert rel_err(data, d) <= TOL_ATOMIC, (dim, size, interp, weights, rel_err(data, d))
                    assert not weights or rel_err(wrec, w) <= TOL_ATOMIC, (dim, size, interp, "weights", rel_err(wrec, w))
                if dim == 3:
                    acc = tp.new_backprojection_accumulator(B, data.shape[-2], "cuda")
                    for _ in range(2):
                        tp.backproject_2d_to_3d_accumulate_interleaved_(acc, c["proj"], c["rot"], c["weights"], c["shifts"], **kw)
                    d2, w2 = tp.fold_backprojection_accumulator(acc)
                    assert rel_err(d2, 2 * d) <= TOL_ATOMIC and rel_err(w2, 2 * w) <= TOL_ATOMIC, (size, interp, "accumulator")
            if os.environ.get("B200PROJ_BRICKS") != "1" and size not in LARGE:      # (brick and slab kernels multiply infinite values by weights of zero)
                check_not_finite(tp, dim, size, {k: v.detach() if v is not None else None for k, v in c.items()})


def check_not_finite(tp, dim, size, c):
    """Infinite and NaN values and weights reach the taps of non-zero weight only; slices with matrices that are not finite, or far
    beyond the box: as from the plain kernels, which run without a workspace and round sample positions alike."""
    B, P, N, _, os_, cutoff = size[:6]
    if P < 9 or N < 8:
        return
    abi = tp._abi
    R = int(abi.load().b200proj_rec_boxsize(N, os_))
    proj, weights, rot, shifts = c["proj"].clone(), c["weights"].clone(), c["rot"].clone(), c["shifts"]
    proj[0, 0, 2, 1] = float("inf")
    proj[0, 3, N - 2, 2] = complex(0.0, float("nan"))
    weights[0, 4, 1, 1] = float("inf")
    rot[0, 5, 0, 0] = float("inf")                      # the samples of a whole slice are nowhere
    rot[0, 6] *= 1e20
    for interp in ("linear", "cubic"):
        code, radius = tp.ops._interp_code(interp), N / 2.0 if cutoff is None else cutoff
        n = abi.load().b200proj_scatter_workspace_bytes(dim, B, P, N, code, 1, os_, radius)
        ws, results = torch.empty(n, dtype=torch.uint8, device="cuda"), []
        for use in (n, 0):
            data = torch.empty((B,) + (R,) * (dim - 1) + (R // 2 + 1,), dtype=torch.complex64, device="cuda")
            wrec = torch.empty(data.shape, device="cuda")
            abi._call("b200proj_backproject_2d_forw" if dim == 2 else "b200proj_backproject_2d_to_3d_forw", proj, proj.data_ptr(), weights.data_ptr(),
                      *abi._geom(B, R, rot, shifts, P, N, code, os_, radius), data.data_ptr(), wrec.data_ptr(), 0, ws.data_ptr() if use else 0, use)
            results.append((torch.view_as_real(data), wrec))
        for a, b in zip(*results):
            ok = torch.isfinite(b)
            assert torch.equal(torch.isfinite(a), ok) and not ok.all(), (dim, size, interp)
            assert (a[ok] - b[ok]).abs().max() <= TOL_ATOMIC * b[ok].abs().max(), (dim, size, interp)


@pytest.mark.parametrize("entries,more", [(0, {"B200PROJ_LIST_SHARED": "4096"}), (3000, {}), (0, {"B200PROJ_LIST_SHARED": "0"}), (3000, {"B200PROJ_LIST_SHARED": "0"}), (0, {"B200PROJ_LIST_CROWD": "100000"}), (3000, {"B200PROJ_LIST_CROWD": "100000", "B200PROJ_BRICKS": "1"})])
def test_cell_sorted_scatters_match_the_oracle(entries, more):
    """entries: of the list; 3,000 make several passes of most sizes.  Few bricks are counted in shared memory; with no such bricks
    all are counted in global memory, as those of reconstructions from about 144^3 on are.  With a limit that no poses reach, the lists are left aside
    and the kernels behind the gate run (the small calls among them are too few pixels for a verdict and keep the lists)."""
    env = dict(os.environ, B200PROJ_LISTS="1", B200PROJ_LIST_ENTRIES=str(entries), **more)
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {str(ROOT / 'tests')!r}); import test_gpu_lists as t; t.check()"],
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("dim,interp,N,P,os_", [(3, "linear", 64, 9000, 1.0), (3, "cubic", 64, 3500, 2.0), (3, "cubic", 96, 900, 1.0), (2, "cubic", 128, 900, 2.0), (2, "linear", 128, 9001, 1.5)])
def test_sizes_that_are_listed_by_themselves_match_double_precision(dim, interp, N, P, os_):
    """Just above the sizes from which lists are chosen: several items per block, weighted and not, several poses in one plane.
    The double-precision kernels do not round sample positions to single precision: up to 4 * 96 * 2^-24 = 2.3e-5 voxels
    apart, times slopes of the taps below 1.3, of random signs."""
    import torch_projectors_b200 as tp
    gen = torch.Generator("cuda").manual_seed(P)
    proj = torch.randn(1, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    w, sh = (torch.rand(s, generator=gen, device="cuda") for s in ((1, P, N, N // 2 + 1), (1, P, 2)))
    sh = sh * 8 - 4
    if dim == 3:
        rot = torch.linalg.qr(torch.randn(1, P, 3, 3, generator=gen, device="cuda"))[0].contiguous()
        rot[:, ::5] = rot[:, :1]
    else:
        a = torch.rand(P, generator=gen, device="cuda") * 6.2832
        rot = torch.stack([a.cos(), -a.sin(), a.sin(), a.cos()], 1).view(1, P, 2, 2)
    code, r = tp.ops._interp_code(interp), N / 2.0
    assert tp._abi.load().b200proj_scatter_workspace_bytes(dim, 1, P, N, code, 1, os_, r) > 4 * 0.7 * P * N * (N // 2 + 1), "not listed"
    forw = tp.backproject_2d_to_3d_forw if dim == 3 else tp.backproject_2d_forw
    kw = dict(interpolation=interp, oversampling=os_)
    d, dw = forw(proj.to(torch.complex128), rot.double(), w.double(), sh.double(), **kw)
    data, wrec = forw(proj, rot, w, sh, **kw)
    assert rel_err(data, d) <= TOL_ATOMIC and rel_err(wrec, dw) <= TOL_ATOMIC
    assert rel_err(forw(proj, rot, None, sh, **kw)[0], d) <= TOL_ATOMIC


@pytest.mark.parametrize("dim,N,os_,P,B,cutoff", [(3, 18, 2.0, 601, 1, None), (3, 6, 1.0, 1501, 2, 4.0), (2, 34, 1.5, 297, 1, 11.5), (2, 66, 1.0, 100, 3, None), (2, 202, 1.0, 1201, 1, None)])
def test_pose_gradients_of_back_projection_by_patches(dim, N, os_, P, B, cutoff):
    """Linear calls of at least 296 slices and 6,000 patches take a slice's patches of 8 x 4 pixels in turn: several blocks to a slice and one, ragged rows and columns, patches
    outside the cutoff, with and without weights and shifts."""
    import torch_projectors_b200 as tp
    from oracle import port
    R = -(-int(N * os_) // 2) * 2
    t = make_inputs(Case("patches", dim, "linear", B, P, N, R, os_, cutoff, 1, 1, shift_range=2.0, seed=N))
    forw, back = (tp.backproject_2d_forw, port.backproject_2d_back) if dim == 2 else (tp.backproject_2d_to_3d_forw, port.backproject_2d_to_3d_back)
    for shifts in (True, False):
        c = {k: v.cuda().requires_grad_(k in ("proj", "weights", "rot", "shifts")) for k, v in t.items()}
        data, wrec = forw(c["proj"], c["rot"], c["weights"], c["shifts"] if shifts else None, interpolation="linear", oversampling=os_, fourier_radius_cutoff=cutoff)
        torch.autograd.backward([data, wrec], [c["grad_data"], c["grad_weight"]])
        want = back(t["grad_data"], t["grad_weight"], t["proj"], t["weights"], t["rot"], t["shifts"] if shifts else None, "linear", os_, cutoff, True, shifts)
        for have, ref, what in zip((c["proj"].grad, c["weights"].grad, c["rot"].grad, c["shifts"].grad if shifts else None), want, ("projections", "weights", "rotations", "shifts")):
            if have is not None:
                assert rel_err(have, ref) <= TOL_ATOMIC, (what, shifts, rel_err(have, ref))


@pytest.mark.parametrize("dim,interp,N,P", [(3, "linear", 64, 9000), (3, "cubic", 48, 4000), (2, "cubic", 128, 900), (2, "linear", 128, 6000)])
def test_a_listed_call_takes_an_infinite_cutoff(dim, interp, N, P):
    """The same as a cutoff beyond the corners of the slices (here: several hundred thousand pixels more than within Nyquist)."""
    import torch_projectors_b200 as tp
    gen = torch.Generator("cuda").manual_seed(P)
    proj = torch.randn(1, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    w = torch.rand(proj.shape, generator=gen, device="cuda")
    rot = torch.linalg.qr(torch.randn(1, P, dim, dim, generator=gen, device="cuda"))[0].contiguous()
    assert tp._abi.load().b200proj_scatter_workspace_bytes(dim, 1, P, N, tp.ops._interp_code(interp), 1, 2.0, float("inf")) > 4 * 0.99 * P * N * (N // 2), "not listed"
    forw = tp.backproject_2d_to_3d_forw if dim == 3 else tp.backproject_2d_forw
    a, aw = forw(proj, rot, w, interpolation=interp, oversampling=2.0, fourier_radius_cutoff=float("inf"))
    b, bw = forw(proj, rot, w, interpolation=interp, oversampling=2.0, fourier_radius_cutoff=float(N))
    assert rel_err(a, b) <= TOL_ATOMIC and rel_err(aw, bw) <= TOL_ATOMIC
    inner, _ = forw(proj, rot, w, interpolation=interp, oversampling=2.0)
    assert rel_err(inner, b) > 100 * TOL_ATOMIC


@pytest.mark.parametrize("P", [167000, 180000])
def test_the_longest_lists(P):
    """Nearly 2^30 entries in one pass (167,000 slices of 128 x 65), and the first number of slices that takes two by itself: the same
    as in parts."""
    import torch_projectors_b200 as tp
    N, gen = 128, torch.Generator("cuda").manual_seed(P)
    inside = tp._abi.cutoff_pack_index(N, N / 2.0, "cuda")[1] - (N // 2)         # (less the mirrored half of column 0)
    assert (inside * P <= 1 << 30) == (P < 170000) and inside * P > 0.99 * (1 << 30)
    proj = torch.randn(1, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    rot = torch.linalg.qr(torch.randn(1, P, 3, 3, generator=gen, device="cuda"))[0].contiguous()
    kw = dict(interpolation="linear", oversampling=1.0)
    whole = tp.backproject_2d_to_3d_forw(proj, rot, None, **kw)[0]
    parts = sum(tp.backproject_2d_to_3d_forw(proj[:, k::3], rot[:, k::3], None, **kw)[0] for k in range(3))
    assert rel_err(whole, parts) <= TOL_ATOMIC


def _one_view(dim, P, gen):
    """Poses that share a plane; in 2D, all slices turned alike."""
    a = torch.rand(P, generator=gen, device="cuda") * 6.2832 if dim == 3 else torch.full((P,), 0.7, device="cuda")
    rot = torch.eye(dim, device="cuda").repeat(P, 1, 1)
    rot[:, 0, 0], rot[:, 0, 1], rot[:, 1, 0], rot[:, 1, 1] = a.cos(), -a.sin(), a.sin(), a.cos()
    return rot


@pytest.mark.parametrize("dim,interp,B,P,N,os_,B_rot", [
    (3, "linear", 1, 9000, 64, 2.0, 1),             # weighted through 16-byte voxels in the workspace, else plain reductions
    (3, "linear", 2, 9000, 50, 2.0, 1),             # poses shared by the batch
    (3, "linear", 1, 500, 352, 1.0, 1),             # volumes taken slab by slab
    (2, "cubic", 2, 800, 64, 2.0, 2), (2, "cubic", 1, 1500, 66, 1.5, 1),
    (2, "linear", 3, 5000, 64, 2.0, 3)])
def test_poses_that_crowd_leave_the_lists_aside(dim, interp, B, P, N, os_, B_rot):
    """Slices of one view run without the lists, uniform poses from them; both as in double precision.  (The verdict is in the
    header: entries listed, pixels found in a brick and in a cell.)"""
    import torch_projectors_b200 as tp
    abi, gen = tp._abi, torch.Generator("cuda").manual_seed(N)
    R = int(abi.rec_boxsize(N, os_))
    code, radius = tp.ops._interp_code(interp), N / 2.0
    proj = torch.randn(B, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    w, sh = torch.rand(proj.shape, generator=gen, device="cuda"), torch.rand(1, P, 2, generator=gen, device="cuda") * 6 - 3
    rec_shape = (B,) + (R,) * (dim - 1) + (R // 2 + 1,)
    n = abi.load().b200proj_scatter_workspace_bytes(dim, B, P, N, code, 1, os_, radius)
    assert n > 0
    for spread in (False, True):
        if spread:
            q = torch.linalg.qr(torch.randn(B_rot, P, dim, dim, generator=gen, device="cuda"))[0]
            rot = (q * torch.linalg.det(q)[..., None, None] if dim == 3 else _turns(B_rot, P, gen)).contiguous()
        else:
            rot = torch.stack([_one_view(dim, P, gen) for _ in range(B_rot)]).contiguous()
        geom = abi._geom(B, R, rot, sh, P, N, code, os_, radius)
        ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
        data, wrec = torch.full(rec_shape, float("nan"), dtype=torch.complex64, device="cuda"), torch.full(rec_shape, float("nan"), device="cuda")
        name = "b200proj_backproject_2d_forw" if dim == 2 else "b200proj_backproject_2d_to_3d_forw"
        abi._call(name, proj, proj.data_ptr(), w.data_ptr(), *geom, data.data_ptr(), wrec.data_ptr(), 0, ws.data_ptr(), n)
        header = ws[:64].view(torch.int32).tolist()
        assert header[9] >= 32 or spread, header
        assert (header[0] > 0) == spread, header
        kw = dict(interpolation=interp, oversampling=os_)
        forw = tp.backproject_2d_to_3d_forw if dim == 3 else tp.backproject_2d_forw
        d, dw = forw(proj.to(torch.complex128), rot.double(), w.double(), sh.double(), **kw)
        assert rel_err(data, d) <= TOL_ATOMIC and rel_err(wrec, dw) <= TOL_ATOMIC, spread
        abi._call(name, proj, proj.data_ptr(), w.data_ptr(), *geom, data.data_ptr(), wrec.data_ptr(), 1, ws.data_ptr(), n)      # adds
        assert rel_err(data, 2 * d) <= TOL_ATOMIC and rel_err(wrec, 2 * dw) <= TOL_ATOMIC, spread
        assert rel_err(forw(proj, rot, None, sh, **kw)[0], d) <= TOL_ATOMIC, spread
        rec = torch.zeros(rec_shape, dtype=torch.complex64, device="cuda")
        back = tp.project_3d_to_2d_back if dim == 3 else tp.project_2d_back
        want = back(proj.to(torch.complex128), rec.to(torch.complex128), rot.double(), sh.double(), **kw)
        assert rel_err(back(proj, rec, rot, sh, **kw), want) <= TOL_ATOMIC, spread
        if dim == 3:
            acc = tp.new_backprojection_accumulator(B, R, "cuda")
            tp.backproject_2d_to_3d_accumulate_interleaved_(acc, proj, rot, w, sh, **kw)
            d2, w2 = tp.fold_backprojection_accumulator(acc)
            assert rel_err(d2, d) <= TOL_ATOMIC and rel_err(w2, dw) <= TOL_ATOMIC, spread


def _turns(B, P, gen):
    a = torch.rand(B, P, generator=gen, device="cuda") * 6.2832
    return torch.stack([a.cos(), -a.sin(), a.sin(), a.cos()], 2).view(B, P, 2, 2)
