"""Entry points with scratch, through the C ABI: a workspace that is missing, too small or off the 16-byte grid is left
alone, the plain kernels run and the results are those with a good one."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from cases import Case, TOL_ATOMIC, TOL_FORWARD, make_inputs, rel_err

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
N, R, OS, P, B = 18, 36, 2.0, 45, 2


def check():
    """In a fresh process with the bricks forced on (the library reads the switch once)."""
    import torch_projectors_b200 as tp
    abi, lib = tp._abi, tp._abi.load()
    for dim in (2, 3):
        t = {k: v.cuda() for k, v in make_inputs(Case("scratch", dim, "cubic", B, P, N, R, OS, None, 1, 1, seed=dim)).items()}
        ptr = {k: v.data_ptr() for k, v in t.items()}
        geom = abi._geom(B, R, t["rot"], t["shifts"], P, N, abi.CUBIC, OS, N / 2.0)
        d, order = ("2d", ()) if dim == 2 else ("3d_to_2d", (0,))
        saving = (f"project_{d}_forw_saving_ws", f"project_{d}_back_saved_ws") if dim == 2 else (f"project_{d}_forw_records", f"project_{d}_back_records")
        back = "backproject_2d_forw" if dim == 2 else "backproject_2d_to_3d_forw"
        n_proj = lib.b200proj_project_workspace_bytes(dim, B, P, N, abi.CUBIC, 1, OS, N / 2.0)
        n_grad = lib.b200proj_gradient_workspace_bytes(dim, B, R, P, N, abi.CUBIC, 0, OS, N / 2.0)
        n_back = lib.b200proj_scatter_workspace_bytes(dim, B, P, N, abi.CUBIC, 1, OS, N / 2.0)
        assert n_proj and n_grad and n_back, "the bricks are not forced on"
        scratch = torch.zeros(max(n_proj, n_grad, n_back) + 64, dtype=torch.uint8, device="cuda")

        def run(kind):
            """All entry points with scratch; kind: good | null | small | off (not on the 16-byte grid)."""
            def ws(n):
                return (scratch.data_ptr() + (8 if kind == "off" else 0) if kind != "null" else 0, n - 1 if kind == "small" else n)
            new = lambda like: torch.full_like(like, float("nan"))  # noqa: E731
            call = lambda name, *args: abi._call("b200proj_" + name, t["rec"], *args)  # noqa: E731
            out, out2, der = new(t["proj"]), new(t["proj"]), torch.zeros((B, P, N, N // 2 + 1, 2 if dim == 2 else 4), dtype=torch.complex64, device="cuda")
            g1, g2, grot, gsh = new(t["rec"]), new(t["rec"]), new(t["rot"]), new(t["shifts"])
            data, wrec = new(t["rec"]), new(t["rec"].real.contiguous())
            call(f"project_{d}_forw_ws", ptr["rec"], *geom, out.data_ptr(), *order, *ws(n_proj))
            call(saving[0], ptr["rec"], *geom, out2.data_ptr(), der.data_ptr(), *order, *ws(n_proj))
            call(f"project_{d}_back_ws", ptr["proj"], ptr["rec"], *geom, g1.data_ptr(), 0, 0, *order, *ws(n_grad))
            call(saving[1], ptr["proj"], out2.data_ptr(), der.data_ptr(), *geom, g2.data_ptr(), grot.data_ptr(), gsh.data_ptr(), *order, *ws(n_grad))
            call(back, ptr["proj"], ptr["weights"], *geom, data.data_ptr(), wrec.data_ptr(), 0, *ws(n_back))
            got = dict(out=out, out2=out2, g1=g1, g2=g2, grot=grot, gsh=gsh, data=data, wrec=wrec)
            if dim == 3:
                got["acc"] = torch.zeros((B, R, R, R // 2 + 1, 4), device="cuda")
                call("backproject_2d_to_3d_accumulate_ws", ptr["proj"], ptr["weights"], *geom, got["acc"].data_ptr(), *ws(n_back))
            torch.cuda.synchronize()
            return got

        want = run("good")
        assert scratch.any(), "a good workspace is used"
        for kind in ("null", "small", "off"):
            scratch.zero_()
            got = run(kind)
            for k, v in got.items():
                assert rel_err(v, want[k]) <= (TOL_FORWARD if k.startswith("out") else TOL_ATOMIC), (dim, kind, k, rel_err(v, want[k]))
            if dim == 3 and kind != "null":
                # (2D: copies of the small reconstruction may use what is aligned but too small for the bricks)
                assert kind == "small" or not scratch.any(), "a misaligned workspace is left alone"


@pytest.mark.parametrize("lists", ["0", "1"])
def test_unusable_scratch_is_left_alone(lists):
    """Without and with pixel lists, in whose place bricks run when the scratch is too small for a list."""
    env = dict(os.environ, B200PROJ_BRICKS="1", B200PROJ_LISTS=lists)
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:0] = [{str(ROOT / 'tests')!r}, {str(ROOT / 'torch-projectors_b200')!r}, {str(ROOT)!r}]; import test_gpu_scratch as t; t.check()"],
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def check_waits():
    """In a fresh process, bricks on and a wait that gives up at its first look: what is lost shows as NaN and in the status word."""
    import torch_projectors_b200 as tp
    abi, lib = tp._abi, tp._abi.load()
    for dim in (2, 3):
        t = {k: v.cuda() for k, v in make_inputs(Case("waits", dim, "cubic", 1, 300, N, R, OS, None, 1, 1, seed=dim)).items()}
        geom = abi._geom(1, R, t["rot"], t["shifts"], 300, N, abi.CUBIC, OS, N / 2.0)
        for weights in (0, 1):
            n = lib.b200proj_scatter_workspace_bytes(dim, 1, 300, N, abi.CUBIC, weights, OS, N / 2.0)
            ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
            data, wrec = torch.zeros_like(t["rec"]), torch.zeros_like(t["rec"].real.contiguous())
            abi._call("b200proj_backproject_2d_forw" if dim == 2 else "b200proj_backproject_2d_to_3d_forw", t["proj"], t["proj"].data_ptr(),
                      t["weights"].data_ptr() if weights else 0, *geom, data.data_ptr(), wrec.data_ptr() if weights else 0, 0, ws.data_ptr(), n)
            torch.cuda.synchronize()
            assert ws[:16].view(torch.int32)[3] == 1
            assert torch.isnan(data.real).any() and (not weights or torch.isnan(wrec).any())
        project = tp.project_3d_to_2d_forw if dim == 3 else tp.project_2d_forw
        rec = t["rec"].requires_grad_(True)
        project(rec, t["rot"], t["shifts"], output_shape=(N, N), interpolation="cubic", oversampling=OS).backward(t["proj"])
        assert torch.isnan(rec.grad.real).any()


def test_a_wait_that_gives_up_shows_in_the_result():
    """With no patience the adding warps' first look at an empty ring ends their wait (the kernel returns by itself)."""
    env = dict(os.environ, B200PROJ_BRICKS="1", B200PROJ_BRICK_WAIT_MS="0")
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:0] = [{str(ROOT / 'tests')!r}, {str(ROOT / 'torch-projectors_b200')!r}, {str(ROOT)!r}]; import test_gpu_scratch as t; t.check_waits()"],
                       env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def check_little_memory():
    """In a fresh process whose allocator may take 60 MB more: cubic scatters whose lists (77 MB) have no room run brick by brick."""
    import ctypes as C
    import torch_projectors_b200 as tp
    lib, P, N = tp._abi.load(), 12000, 64
    gen = torch.Generator("cuda").manual_seed(0)
    proj = torch.randn(1, P, N, N // 2 + 1, dtype=torch.complex64, generator=gen, device="cuda")
    w, rot = torch.rand(proj.shape, generator=gen, device="cuda"), torch.linalg.qr(torch.randn(1, P, 3, 3, generator=gen, device="cuda"))[0].contiguous()
    rec = torch.zeros(1, 2 * N, 2 * N, N + 1, dtype=torch.complex64, device="cuda")
    acc = tp.new_backprojection_accumulator(1, 2 * N, "cuda")
    kw = dict(interpolation="cubic", oversampling=2.0)
    none = C.c_size_t(-1).value
    calls = {"weighted": lambda: tp.backproject_2d_to_3d_forw(proj, rot, w, **kw), "plain": lambda: tp.backproject_2d_to_3d_forw(proj, rot, None, **kw)[0],
             "gradient": lambda: tp.project_3d_to_2d_back(proj, rec, rot, **kw),
             "accumulator": lambda: tp.backproject_2d_to_3d_accumulate_interleaved_(acc.zero_(), proj, rot, w, **kw) or acc}
    want = {k: f() for k, f in calls.items()}
    want["accumulator"] = acc.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (60 << 20)) / total)
    for k, f in calls.items():
        mode = {"weighted": 1, "plain": 0, "gradient": 0, "accumulator": 2}[k]
        sizes = [lib.b200proj_scatter_workspace_bytes_within(3, 1, P, N, tp._abi.CUBIC, mode, 2.0, N / 2.0, most) for most in (none, 60 << 20)]
        assert sizes[0] > 77e6 > 20e6 > sizes[1] > 0, sizes
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        got = f()
        torch.cuda.synchronize()
        outputs = torch.cuda.memory_allocated() - before
        scratch = torch.cuda.max_memory_allocated() - before - outputs
        assert scratch >= sizes[1], (k, scratch, sizes)
        for a, b in zip(got if isinstance(got, tuple) else (got,), want[k] if isinstance(want[k], tuple) else (want[k],)):
            assert rel_err(a, b) <= TOL_ATOMIC, (k, rel_err(a, b))
        del got


def test_scatters_without_room_for_lists_take_the_next_smaller_scratch():
    r = subprocess.run([sys.executable, "-c", f"import sys; sys.path[:0] = [{str(ROOT / 'tests')!r}, {str(ROOT / 'torch-projectors_b200')!r}, {str(ROOT)!r}]; import test_gpu_scratch as t; t.check_little_memory()"],
                       cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
