"""The brick-by-brick 3D kernels (a block keeps a piece of the volume in shared memory and walks over the slices)
against the CPU oracle, at sizes and poses where the walk can go wrong: one brick and several, ragged boxes and pose
counts, lattice poses, matrices that are no rotations, cutoffs inside and beyond Nyquist, batches."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from cases import Case, TOL_ATOMIC, TOL_FORWARD, axis_aligned_rotations, make_inputs, random_rotations_2d, random_rotations_3d, rel_err

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

#      B  P   N   R   os    cutoff  B_rot  B_shift
SIZES = [(1, 40, 4, 8, 2.0, None, 1, 1),
         (1, 45, 18, 36, 2.0, None, 1, 1),
         (2, 33, 20, 30, 1.5, 7.3, 2, 0),
         (2, 9, 34, 34, 1.0, 20.0, 1, 2),
         (1, 37, 26, 34, 1.3, None, 1, 1),
         (1, 3, 48, 120, 2.5, 17.0, 1, 1),
         (1, 12, 44, 100, 2.0, 29.0, 1, 1)]          # cutoff beyond Nyquist: corners of the slices


SIZES_2D = SIZES[:5] + [(1, 21, 70, 160, 2.0, 40.0, 1, 1), (2, 300, 130, 130, 1.0, None, 2, 2)]


def _inputs(dim, size, seed):
    B, P, N, R, os_, cutoff, B_rot, B_shift = size
    t = make_inputs(Case("bricks", dim, "cubic", B, P, N, R, os_, cutoff, B_rot, B_shift, shift_range=5.0, seed=seed))
    lattice = axis_aligned_rotations(torch.Generator().manual_seed(seed))
    if dim == 2:
        t["rot"][0, 3] *= 1.2
        lattice = t["rot"][0, :1].repeat(P + 1, 1, 1)
    if P >= len(lattice):
        t["rot"][0, : len(lattice)] = lattice
        t["rot"][0, len(lattice)] *= 1.2                    # not rotations: these slices take the plain path
    if P > 2:
        t["rot"][0, 2, :, 1] = t["rot"][0, 2, :, 0]
    return t, dict(output_shape=(N, N), oversampling=os_, fourier_radius_cutoff=cutoff)


def check(names):
    """Run in a fresh process with the bricks forced on (the library reads the switch once)."""
    for dim in (3, 2):
        check_dim(names, dim)


def check_dim(names, dim):
    sys.path[:0] = [str(ROOT), str(ROOT / "torch-projectors_b200"), str(ROOT / "tests")]
    import torch_projectors_b200 as tp
    from oracle import port
    project, reference, gradient = ((tp.project_3d_to_2d_forw, port.project_3d_to_2d_forw, port.project_3d_to_2d_back) if dim == 3 else
                                    (tp.project_2d_forw, port.project_2d_forw, port.project_2d_back))
    backproject, back_reference = ((tp.backproject_2d_to_3d_forw, port.backproject_2d_to_3d_forw) if dim == 3 else
                                   (tp.backproject_2d_forw, port.backproject_2d_forw))
    for seed, size in enumerate(SIZES if dim == 3 else SIZES_2D):
        for interp in ("linear", "cubic"):
            t, kw = _inputs(dim, size, seed)
            N, os_, cutoff = size[2], size[4], size[5]
            want = reference(t["rec"], t["rot"], t["shifts"], [N, N], interp, os_, cutoff)
            sizes = (dim, size[0], size[1], N, tp.ops._interp_code(interp))
            lib, radius = tp._abi.load(), N / 2.0 if cutoff is None else cutoff
            assert (interp == "linear" and dim == 2) or lib.b200proj_project_workspace_bytes(*sizes, 0, os_, radius) > 0, "the bricks are not forced on"
            assert interp == "linear" or all(lib.b200proj_scatter_workspace_bytes(*sizes, w, os_, radius) > 0 for w in (0, 1))
            shifts = t["shifts"].cuda() if t["shifts"] is not None else None
            if "forward" in names:
                got = project(t["rec"].cuda(), t["rot"].cuda(), shifts, interpolation=interp, **kw)
                assert rel_err(got, want) <= TOL_FORWARD, (size, interp, rel_err(got, want))
            if "gradients" in names:
                tp.set_save_derivatives(True, min_volume_bytes=0)
                for fixed in (False, True):
                    rec, rot = t["rec"].cuda().requires_grad_(not fixed), t["rot"].cuda().requires_grad_(True)
                    sh = shifts.clone().requires_grad_(True) if shifts is not None else None
                    out = project(rec, rot, sh, interpolation=interp, **kw)
                    assert rel_err(out, want) <= TOL_FORWARD, (size, interp)
                    out.backward(t["proj"].cuda())
                    grads = gradient(t["proj"], t["rec"], t["rot"], t["shifts"], interp, os_, cutoff,
                                                       need_rot_grad=True, need_shift_grad=shifts is not None)
                    for have, ref, what in ((rec.grad, grads[0], "volume"), (rot.grad, grads[1], "rotations"), (sh.grad if sh is not None else None, grads[2], "shifts")):
                        if have is not None:
                            assert rel_err(have, ref) <= TOL_ATOMIC, (size, interp, what, rel_err(have, ref))
                rec = t["rec"].cuda().requires_grad_(True)                 # the volume's gradient alone
                project(rec, t["rot"].cuda(), shifts, interpolation=interp, **kw).backward(t["proj"].cuda())
                assert rel_err(rec.grad, grads[0]) <= TOL_ATOMIC, (size, interp, "volume alone")
            if "backprojection" in names:
                for weights in (None, t["weights"]):
                    data, wrec = backproject(t["proj"].cuda(), t["rot"].cuda(), weights.cuda() if weights is not None else None, shifts,
                                                              interpolation=interp, oversampling=os_, fourier_radius_cutoff=cutoff)
                    ref, wref = back_reference(t["proj"], weights, t["rot"], t["shifts"], interp, os_, cutoff)
                    assert rel_err(data, ref) <= TOL_ATOMIC, (size, interp, "data", rel_err(data, ref))
                    if weights is not None and dim == 3:
                        acc = tp.new_backprojection_accumulator(size[0], data.shape[-2], "cuda")
                        tp.backproject_2d_to_3d_accumulate_interleaved_(acc, t["proj"].cuda(), t["rot"].cuda(), weights.cuda(), shifts,
                                                                        interpolation=interp, oversampling=os_, fourier_radius_cutoff=cutoff)
                        d2, w2 = tp.fold_backprojection_accumulator(acc)
                        assert rel_err(d2, ref) <= TOL_ATOMIC and rel_err(w2, wref) <= TOL_ATOMIC, (size, interp, "accumulator")
                    if weights is not None:
                        assert rel_err(wrec, wref) <= TOL_ATOMIC, (size, interp, "weights", rel_err(wrec, wref))


@pytest.mark.parametrize("names", ["forward", "gradients", "backprojection"])
def test_bricks_match_the_oracle(names):
    env = dict(os.environ, B200PROJ_BRICKS="1")
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {str(ROOT / 'tests')!r}); import test_gpu_bricks as t; t.check({names!r})"],
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("dim,interp,P", [(2, "linear", 64), (2, "cubic", 67), (3, "linear", 130), (2, "cubic", 63)])
def test_scatters_spread_over_copies_of_a_small_reconstruction(dim, interp, P):
    """From 64 poses on, slices are spread over copies of a small reconstruction that are added up at the end: gradients
    (with and without pose gradients) and back-projection without weights, against the oracle."""
    import torch_projectors_b200 as tp
    from oracle import port
    t = make_inputs(Case("copies", dim, interp, 2, P, 12, 18, 1.5, None, 1, 2, shift_range=2.0, seed=P))
    project, back = (tp.project_2d_forw, port.project_2d_back) if dim == 2 else (tp.project_3d_to_2d_forw, port.project_3d_to_2d_back)
    want = back(t["proj"], t["rec"], t["rot"], t["shifts"], interp, 1.5, None, need_rot_grad=True, need_shift_grad=True)
    for poses in (True, False):
        for keep in (True, False):
            tp.set_save_derivatives(keep, min_volume_bytes=0)
            try:
                rec, rot, sh = (t[k].cuda().requires_grad_(k == "rec" or poses) for k in ("rec", "rot", "shifts"))
                project(rec, rot, sh, output_shape=(12, 12), interpolation=interp, oversampling=1.5).backward(t["proj"].cuda())
            finally:
                tp.set_save_derivatives(True)
            assert rel_err(rec.grad, want[0]) <= TOL_ATOMIC
            if poses:
                assert rel_err(rot.grad, want[1]) <= TOL_ATOMIC and rel_err(sh.grad, want[2]) <= TOL_ATOMIC
    forw, ref = (tp.backproject_2d_forw, port.backproject_2d_forw) if dim == 2 else (tp.backproject_2d_to_3d_forw, port.backproject_2d_to_3d_forw)
    data, _ = forw(t["proj"].cuda(), t["rot"].cuda(), None, t["shifts"].cuda(), interpolation=interp, oversampling=1.5)
    assert rel_err(data, ref(t["proj"], None, t["rot"], t["shifts"], interp, 1.5, None)[0]) <= TOL_ATOMIC


def _matrices(dim, size, seed):
    """Poses that are no rotations: magnified (up to and beyond what bricks take), sheared, mirrored, slightly perturbed, singular."""
    B, P, N, R, os_, cutoff, B_rot, B_shift = size
    t = make_inputs(Case("matrices", dim, "cubic", B, P, N, R, os_, cutoff, B_rot, B_shift, shift_range=5.0, seed=seed))
    gen = torch.Generator().manual_seed(seed)
    for p in range(P):
        m = t["rot"][:, p]
        kind = p % 8
        if kind == 0:
            m *= (0.05, 0.12, 0.3, 0.7, 1.01, 1.08, 1.3, 1.7, 2.0, 2.3)[p // 8 % 10]
        elif kind == 1:
            m += 0.02 * torch.randn(m.shape, generator=gen)
        elif kind == 2:
            m[..., 1] += (0.3, 1.0, 4.0)[p // 8 % 3] * m[..., 0]
        elif kind == 3:
            m[..., 0] *= -1.0
        elif kind == 4:
            m *= torch.tensor([1.25, 0.8, 1.0][:dim])
        elif kind == 5:
            m *= 0.0 if p // 8 % 2 else 1.0 + 1e-4
    return t, dict(output_shape=(N, N), oversampling=os_, fourier_radius_cutoff=cutoff)


def check_matrices(names):
    global _inputs, SIZES, SIZES_2D
    _inputs = _matrices
    SIZES = [(1, 100, 18, 36, 2.0, None, 1, 1), (2, 83, 34, 50, 1.5, 13.0, 1, 2), (1, 80, 20, 20, 1.0, 14.0, 1, 0)]
    SIZES_2D = SIZES + [(1, 90, 70, 160, 2.0, 40.0, 1, 1)]
    check(names)


@pytest.mark.parametrize("names", ["forward", "gradients", "backprojection"])
def test_bricks_match_the_oracle_for_matrices_that_are_no_rotations(names):
    env = dict(os.environ, B200PROJ_BRICKS="1")
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {str(ROOT / 'tests')!r}); import test_gpu_bricks as t; t.check_matrices({names!r})"],
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("dim,interp,P,copies", [(2, "linear", 4000, 32), (2, "cubic", 1031, 32), (3, "linear", 1501, 32), (3, "cubic", 257, 8), (3, "cubic", 20, 1)])
def test_scatters_choose_copies_by_the_reductions_per_byte(dim, interp, P, copies):
    """At sizes where the copies are chosen by themselves (many slices onto a small reconstruction), and where not:
    gradients with and without pose gradients and back-projection without weights, against the oracle."""
    import torch_projectors_b200 as tp
    from oracle import port
    t = make_inputs(Case("copies", dim, interp, 1, P, 12, 18, 1.5, None, 1, 1, shift_range=2.0, seed=P))
    one = 8 * (18 if dim == 3 else 1) * 18 * 10
    have = tp._abi.load().b200proj_gradient_workspace_bytes(dim, 1, 18, P, 12, tp.ops._interp_code(interp), 0, 1.5, 6.0)
    assert have == (copies * one if copies > 1 else 0)
    project, back = (tp.project_2d_forw, port.project_2d_back) if dim == 2 else (tp.project_3d_to_2d_forw, port.project_3d_to_2d_back)
    want = back(t["proj"], t["rec"], t["rot"], t["shifts"], interp, 1.5, None, need_rot_grad=True, need_shift_grad=True)
    for poses in (True, False):
        rec, rot, sh = (t[k].cuda().requires_grad_(k == "rec" or poses) for k in ("rec", "rot", "shifts"))
        project(rec, rot, sh, output_shape=(12, 12), interpolation=interp, oversampling=1.5).backward(t["proj"].cuda())
        assert rel_err(rec.grad, want[0]) <= TOL_ATOMIC
        if poses:
            assert rel_err(rot.grad, want[1]) <= TOL_ATOMIC and rel_err(sh.grad, want[2]) <= TOL_ATOMIC
    forw, ref = (tp.backproject_2d_forw, port.backproject_2d_forw) if dim == 2 else (tp.backproject_2d_to_3d_forw, port.backproject_2d_to_3d_forw)
    data, _ = forw(t["proj"].cuda(), t["rot"].cuda(), None, t["shifts"].cuda(), interpolation=interp, oversampling=1.5)
    assert rel_err(data, ref(t["proj"], None, t["rot"], t["shifts"], interp, 1.5, None)[0]) <= TOL_ATOMIC


def _one_plane(t, share):
    """Every `share`-th pose becomes an in-plane turn of one and the same plane: a few bricks get all of its pixels."""
    turns = torch.linspace(0, 6.2, t["rot"][:, ::share].shape[1])
    t["rot"][:, ::share, :2, :2] = torch.stack([turns.cos(), -turns.sin(), turns.sin(), turns.cos()], 1).view(1, -1, 2, 2)
    t["rot"][:, ::share, 2] = torch.tensor([0.0, 0.0, 1.0])
    t["rot"][:, ::share, :, 2] = torch.tensor([0.0, 0.0, 1.0])


@pytest.mark.parametrize("os_,P,share", [(2.0, 3000, 1), (2.0, 3001, 3), (1.0, 2999, 2)])
def test_scatters_that_run_in_bricks_by_themselves_match_the_oracle(os_, P, share):
    """Cubic 3D calls just above the sizes from which bricks are chosen: several items per brick and per block."""
    import torch_projectors_b200 as tp
    from oracle import port
    N, R = 32, int(32 * os_)
    t = make_inputs(Case("rings", 3, "cubic", 1, P, N, R, os_, None, 1, 1, shift_range=4.0, seed=P, special_poses=False))
    _one_plane(t, share)
    lib, cubic = tp._abi.load(), tp._abi.CUBIC
    assert all(lib.b200proj_scatter_workspace_bytes(3, 1, P, N, cubic, w, os_, N / 2.0) > 0 for w in (0, 1))
    c = {k: v.cuda() for k, v in t.items()}
    kw = dict(interpolation="cubic", oversampling=os_)
    got = tp.project_3d_to_2d_back(c["proj"], c["rec"], c["rot"], c["shifts"], **kw)
    assert rel_err(got, port.project_3d_to_2d_back(t["proj"], t["rec"], t["rot"], t["shifts"], "cubic", os_, None)[0]) <= TOL_ATOMIC
    for weights in (None, "weights"):
        data, wrec = tp.backproject_2d_to_3d_forw(c["proj"], c["rot"], c[weights] if weights else None, c["shifts"], **kw)
        ref, wref = port.backproject_2d_to_3d_forw(t["proj"], t[weights] if weights else None, t["rot"], t["shifts"], "cubic", os_, None)
        assert rel_err(data, ref) <= TOL_ATOMIC and (weights is None or rel_err(wrec, wref) <= TOL_ATOMIC)


LONG_RUNS = [(3, 64, 12000), (3, 80, 7919), (2, 128, 3001)]


def check_long_runs(dim, N, P, lists):
    """Against the double-precision kernels (which run neither in bricks nor from lists).  Their sample positions are not rounded to
    single precision: up to 4 * 160 * 2^-24 = 4e-5 voxels apart, times slopes of the taps below 1.3, of random signs."""
    import torch_projectors_b200 as tp
    lib, cubic = tp._abi.load(), tp._abi.CUBIC
    gen = torch.Generator("cuda").manual_seed(N)
    real = lambda *s: torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    proj = torch.randn(1, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    w, sh = real(1, P, N, N // 2 + 1), real(1, P, 2) * 8 - 4
    rot = {"rot": (random_rotations_3d if dim == 3 else random_rotations_2d)(P, torch.Generator().manual_seed(N)).view(1, P, dim, dim)}
    if dim == 3:
        _one_plane(rot, 3)
    rot = rot["rot"].cuda()
    # a list holds every pixel within Nyquist (0.39 N^2 a slice), bricks hold records of the slices
    sizes = [lib.b200proj_scatter_workspace_bytes(dim, 1, P, N, cubic, k, 2.0, N / 2.0) for k in (0, 1)]
    assert all(n > 0 and (n > 4 * 0.39 * P * N * N) == lists for n in sizes), sizes
    forw = tp.backproject_2d_to_3d_forw if dim == 3 else tp.backproject_2d_forw
    back = tp.project_3d_to_2d_back if dim == 3 else tp.project_2d_back
    kw = dict(interpolation="cubic", oversampling=2.0)
    d, dw = forw(proj.to(torch.complex128), rot.double(), w.double(), sh.double(), **kw)
    data, wrec = forw(proj, rot, w, sh, **kw)
    assert rel_err(data, d) <= TOL_ATOMIC and rel_err(wrec, dw) <= TOL_ATOMIC
    assert rel_err(forw(proj, rot, None, sh, **kw)[0], d) <= TOL_ATOMIC
    rec = torch.zeros_like(data)
    assert rel_err(back(proj, rec, rot, sh, **kw), back(proj.to(torch.complex128), rec.to(torch.complex128), rot.double(), sh.double(), **kw)) <= TOL_ATOMIC
    if dim == 3:
        acc = tp.new_backprojection_accumulator(1, 2 * N, "cuda")
        tp.backproject_2d_to_3d_accumulate_interleaved_(acc, proj, rot, w, sh, **kw)
        d2, w2 = tp.fold_backprojection_accumulator(acc)
        assert rel_err(d2, d) <= TOL_ATOMIC and rel_err(w2, dw) <= TOL_ATOMIC


@pytest.mark.parametrize("dim,N,P", LONG_RUNS)
def test_long_runs_of_the_scatter_rings_match_double_precision(dim, N, P):
    """Enough slices that a walking warp refills its list of hits and rings and sums are used over many items of a block.  In a
    process of its own: calls of this size run from pixel lists unless these are off."""
    code = f"import sys; sys.path[:0] = [{str(ROOT / 'tests')!r}, {str(ROOT / 'torch-projectors_b200')!r}, {str(ROOT)!r}]; import test_gpu_bricks as t; t.check_long_runs({dim}, {N}, {P}, False)"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, B200PROJ_LISTS="0"), cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("dim,N,P", LONG_RUNS)
def test_the_same_from_pixel_lists(dim, N, P):
    check_long_runs(dim, N, P, True)
