"""Memory safety of the kernels that the small grids of test_gpu_bounds.py do
not reach by whole steps, in the bounds-checked library (MW_CHECK=1): single
stages of every form (the FP32 ones from tensor copies and from plain loads, the
x stage's kernel for short rows), steps of grids above each limit of the line
kernels (launches that overlap; the FP32 direction kernels with four and eight
cells a lane, with the forcing, over one and many tiles), the host-buffer step
in several ragged bands, the adjoint's tiles of every width, solution variables
in pieces and in blocks of rows, ensembles whose z tiles are cut."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = textwrap.dedent("""
    import ctypes, torch
    from pyminiweather_gb300 import _native
    from pyminiweather_gb300.data import initialize_fields
    from pyminiweather_gb300.ensemble import Ensemble, member_params
    from pyminiweather_gb300.ics import init
    from pyminiweather_gb300.post import compute_stats, compute_solution_variables
    from pyminiweather_gb300.solve import evolve, evolve_host, reset_direction
    from tests.helpers import make_params
    L = _native.load()
    assert _native.library_path().endswith("_check.so"), _native.library_path()
    n = ctypes.c_ulonglong(0)
    S = _native.stream_handle()
    P = _native.ptr
    MODES = _native.F64_MODES
    def count(*what):
        torch.cuda.synchronize()
        _native.call("mw_debug_oob_count", ctypes.byref(n), 0)
        print(*what, "OOB so far", n.value, flush=True)
    def fields(p, dtype=torch.float64):
        f = initialize_fields(p, dtype=dtype)
        init(f, p, None)
        reset_direction()
        return f
    _native.call("mw_debug_oob_count", ctypes.byref(n), 1)
    t = ctypes.c_ulonglong(1)
    _native.call("mw_debug_wait_timeouts", ctypes.byref(t), 1)
    # single stages: nx % 4 == 0 and nx >= 128 take tensor copies in FP32
    for nx, nz, ic in [(2, 1, "thermal"), (3, 700, "thermal"), (2, 21001, "thermal"), (30, 5001, "collision"),
                       (31, 5, "gravity"), (62, 17, "collision"), (66, 1301, "gravity"), (94, 33, "thermal"),
                       (130, 70, "gravity"), (257, 129, "collision"), (2047, 66, "collision"), (4000, 16, "gravity"),
                       (128, 33, "gravity"), (132, 7, "collision"), (256, 64, "thermal"), (260, 9, "gravity"),
                       (1024, 130, "collision")]:
        p = make_params(nx, nz, ic)
        for dtype in (torch.float64, torch.float32):
            f = fields(p, dtype)
            hb = [P(a) for a in f.backgrounds()]
            frc, out = f.state.clone(), torch.empty_like(f.state)
            for direction in (0, 1):
                for flags in (0, 1):
                    args = (nx, nz, p["dx"], p["dz"], p["dt"], *hb, P(f.src_w), P(f.state), P(frc), P(out),
                            p["dt"] / 2, direction)
                    if dtype == torch.float32:
                        _native.call("mw_dirstage_f32", *args, flags, S)
                    else:
                        for mode in (0, 1, 2):
                            _native.call("mw_dirstage_f64", *args, mode, flags, S)
        count("stages", nx, nz)
    # steps above the line kernels' limits
    for nx, nz, ic, forms in [(1001, 301, "gravity", "f"), (1001, 301, "collision", "f"), (8, 40001, "gravity", "fi"),
                              (16100, 9, "gravity", "f"), (20000, 2, "collision", "f"), (20000, 1, "gravity", "f"),
                              (1001, 601, "gravity", "is"), (1203, 500, "collision", "is"), (5000, 13, "gravity", "s"),
                              (13, 5000, "collision", "s"), (2, 70001, "thermal", "is"), (100001, 3, "gravity", "ifs")]:
        for form, dtype, mode in (("f", torch.float32, "fp64"), ("i", torch.float64, "fp64"), ("s", torch.float64, "split")):
            if form not in forms:
                continue
            for flags in (1, 0):
                p = dict(make_params(nx, nz, ic), f64_mode=mode, step_flags=flags)
                f = fields(p, dtype)
                evolve(p, f, None, dt=p["dt"], nsteps=2)
                evolve(p, f, None, dt=p["dt"], nsteps=1)
        count("steps", nx, nz, ic, forms)
    # the host-buffer step in bands
    for nx, nz, nbands, want, ic in [(2050, 1031, 3, 3, "gravity"), (3001, 1751, 10, 10, "collision")]:
        for mode in ("fp64", "split"):
            assert L.mw_host_step_bands(nx, nz, MODES[mode], nbands) == want
            for flags in (1, 0):
                p = dict(make_params(nx, nz, ic), f64_mode=mode, step_flags=flags, check_finite=True)
                f = fields(p)
                h = f.state.cpu().pin_memory()
                evolve_host(p, f, h, h, dt=p["dt"], nbands=nbands)
                evolve_host(p, f, h, h, dt=p["dt"], nbands=nbands)
        count("host", nx, nz, nbands)
    # the adjoint's tiles
    for nx, nz in [(2, 1), (2, 3), (2, 509), (2, 1021), (3, 1100), (5, 70), (8, 125), (9, 126), (16, 61), (17, 62),
                   (66, 900), (255, 200), (4000, 1), (3001, 2), (3001, 5), (3000, 7), (3000, 8), (512, 60)]:
        p = make_params(nx, nz, "collision")
        f = fields(p)
        hb = [P(a) for a in f.backgrounds()]
        ws = torch.empty(int(L.mw_dirstage_vjp_workspace_bytes(nx, nz)) // 8 + 1, dtype=torch.float64, device="cuda")
        g, out = torch.randn_like(f.state), torch.empty_like(f.state)
        for mode in (0, 1, 2):
            for d in (0, 1):
                _native.call("mw_dirstage_vjp_f64", nx, nz, p["dx"], p["dz"], p["dt"], *hb, P(f.state), P(g), P(g),
                             None, 1, P(out), p["dt"] / 3, d, mode, P(ws), ws.numel() * 8, S)
        count("adjoint", nx, nz)
    for nx, nz in [(2, 1), (3, 1000), (7, 5000), (100, 1000), (683, 700), (1024, 700), (257, 3), (2049, 5), (40961, 9),
                   (20000, 2)]:
        p = make_params(nx, nz, "collision")
        f = fields(p)
        compute_solution_variables(p, f)
        compute_stats(p, f)
    count("diagnostics")
    for sizes in ([(130, 70), (64, 33), (65, 129), (2, 1)], [(100, 50)] * 30, [(300, 40)]):
        for dtype, mode in ((torch.float64, "fp64"), (torch.float64, "split"), (torch.float32, "fp64")):
            for z_tile in (5, 16, 64):
                ens = Ensemble([(member_params(a, b), None) for a, b in sizes], dtype=dtype, f64_mode=mode,
                               z_tile=z_tile)
                ens.step(3)
    count("ensembles")
    assert n.value == 0, n.value
    print("OOB 0 in all")
    _native.call("mw_debug_wait_timeouts", ctypes.byref(t), 0)
    assert t.value == 0, t.value  # of the tensor-copy stages above
""")


def test_stages_and_large_grids_stay_in_bounds():
    env = dict(os.environ, MW_LIBRARY_VARIANT="check",
               PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", DRIVER], cwd=ROOT, capture_output=True, text=True, timeout=1500, env=env)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-4000:])
    assert "OOB 0 in all" in r.stdout
