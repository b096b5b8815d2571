"""The Jacobi-PCG loops of the heat solver at the edges of their kernels: the
one-kernel loop (tiles of 128 x 2 cells, 1, 2, 4 or 8 of them a CTA, one CTA an
SM) and the two-kernel loop beyond it (strips of 30 columns), FP64 and
mixed. Held to the FP64 residual recomputed by numpy and, as far as the two
residuals allow them to differ, to the solution of the flexible CG with
Jacobi (other kernels, the same solve)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def residual(Kx, Ky, u, u0, rx):
    c, e, n = (slice(1, -1), slice(1, -1)), (slice(1, -1), slice(2, None)), (slice(2, None), slice(1, -1))
    w, s = (slice(1, -1), slice(None, -2)), (slice(None, -2), slice(1, -1))
    return u0[c] - ((1.0 + rx * (Ky[n] + Ky[c] + Kx[e] + Kx[c])) * u[c] - rx * (Ky[n] * u[n] + Ky[c] * u[s])
                    - rx * (Kx[e] * u[e] + Kx[c] * u[w]))


def one_kernel(nx, ny):
    """Whether the grid's tiles fit one CTA an SM, 8 to a CTA at most."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gx, gy = -(-nx // 128), -(-ny // 2)
    return gx * gy <= 1184 and any(gx * -(-gy // k) <= sms for k in (1, 2, 4, 8))


# nx, ny: one cell; a tile's last column and the next CTA's first; 1, 2, 4 and 8
# tiles a CTA, with ragged ends; on 148 SMs the tallest grid of the one-kernel
# loop 8 tiles wide (8 x 144) and the first beyond it; strips of 30, 31 and 61
# columns; more strips than 4096 CTAs hold
@pytest.mark.parametrize("nx,ny", [(1, 1), (128, 2), (129, 3), (127, 33), (61, 600), (257, 301), (1024, 296),
                                   (1024, 298), (31, 2400), (150, 1190), (1230, 61), (990001, 2), (256, 192),
                                   (500, 511), (1024, 288), (1024, 290)])
@pytest.mark.parametrize("method", ["PCG_TRUE", "PCG", "MIXED"])
def test_loops_reach_the_residual(gpu_runtime, nx, ny, method):
    import torch

    from ops_b200 import lmg
    rng = np.random.default_rng(nx * 7 + ny)
    rho = np.exp(rng.uniform(np.log(0.1), np.log(10.0), (ny, nx)))
    Kx, Ky, u0 = lmg.padded_problem(rho, rng.uniform(0.0, 1.0, (ny, nx)))
    # open edges too: a non-zero boundary face next to the ring's zero
    Kx[1:-1, 1] = Kx[1:-1, -1] = 0.3
    k = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (Kx, Ky, u0)]
    u, v = k[2].clone(), k[2].clone()
    u[0], u[-1], u[:, 0], u[:, -1] = 0.0, 0.0, 0.0, 0.0
    v.copy_(u)
    st = lmg.solve(*k, u, 20.0, 20.0, method=getattr(lmg, method), eps=1e-10)
    ref = lmg.solve(*k, v, 20.0, 20.0, method=lmg.FCG_JACOBI, eps=1e-12)
    assert st["converged"] and ref["converged"]
    # the one-kernel loop is one launch, between the set-up's two and the residual (mixed: for each
    # update the restart, the loop, the update and the residual); a chunk of the other loop is 32
    whole = 2 + 4 * st["updates"] if method == "MIXED" else 4
    assert st["launches"] == whole if one_kernel(nx, ny) else st["launches"] >= whole + 31
    a, b = u.cpu().numpy(), v.cpu().numpy()
    r = np.linalg.norm(residual(Kx, Ky, a, u0, 20.0))
    # PCG stops on sqrt|r.z| < eps ||r0|| (TeaLeaf's rule), so ||r|| < sqrt(max D) eps ||r0|| with
    # D <= 1 + 20 * 4 * 10 (faces are at most 1 / 0.1): a factor of 28.3
    bound = (1.5 if method != "PCG" else 30.0) * 1e-10 * st["initial_residual"]
    assert r <= max(bound, 1e-13 * np.linalg.norm(u0)), (r, bound)
    # A is the identity plus a positive semidefinite operator: ||u - v|| <= ||A (u - v)||
    s = np.linalg.norm(residual(Kx, Ky, b, u0, 20.0))
    assert np.linalg.norm(a - b) <= r + s + 1e-12 * np.linalg.norm(b)
    if method == "PCG_TRUE" and ref["iterations"] > 3:
        assert st["iterations"] < ref["iterations"]


@pytest.mark.parametrize("method", ["PCG_TRUE", "MIXED"])
def test_wide_cross_section_3d(gpu_runtime, method):
    """A cross-section of more than 4096 tiles."""
    import torch

    from ops_b200 import lmg
    rng = np.random.default_rng(5)
    rho = np.exp(rng.uniform(np.log(0.1), np.log(10.0), (2, 1400, 1400)))
    k = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in lmg.faces3d(rho)]
    u0 = torch.zeros_like(k[0])
    u0[1:-1, 1:-1, 1:-1] = torch.from_numpy(rng.uniform(0.0, 1.0, rho.shape)).cuda()
    u = u0.clone()
    st = lmg.solve3d(*k, u0, u, 5.0, 5.0, 5.0, method=getattr(lmg, method), eps=1e-8)
    # stopped on the recursive residual (PCG_TRUE) or the FP64 one; they differ by rounding, far below 1e-8 ||r0||
    assert st["converged"] and st["final_residual"] < 1.5e-8 * st["initial_residual"]


@pytest.mark.parametrize("method", ["PCG_TRUE", "FCG_JACOBI", "FCG_MG"])
def test_second_direction_takes_no_field_of_its_own(gpu_runtime, method):
    """The solver's own fields are six (and the multigrid levels): the second
    direction goes to one of them. In a process of its own, for the fields
    outlive a solve."""
    import subprocess
    import sys
    code = f"""
import numpy as np, torch
from ops_b200 import lmg
def solve(n):
    rho = np.ones((n, n))
    en = np.random.default_rng(1).random((n, n))
    k = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in lmg.padded_problem(rho, en)]
    u = k[2].clone()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    lmg.solve(*k, u, 20.0, 20.0, method=lmg.{method}, eps=1e-8)
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0]
solve(640)
field = 8 * 2050 ** 2
levels = 4 * 6 * 2080 * 2048 * 4 / 3 if {method!r} == "FCG_MG" else 0
kept = solve(2048) + 6 * 8 * 642 ** 2
assert kept < 6.5 * field + levels, (kept, field)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("method", ["PCG_TRUE", "MIXED"])
def test_expired_wait_is_an_error_and_the_solver_goes_on(gpu_runtime, method):
    """No wait of the one-kernel loop may succeed (heat_wait_ms 0): the solve
    ends with a timeout, leaves u as it was, and the next one is as ever."""
    import torch

    from ops_b200 import _lib, lmg
    from ops_b200 import ops as O
    rng = np.random.default_rng(3)
    rho = np.exp(rng.uniform(np.log(0.1), np.log(10.0), (140, 300)))
    k = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in lmg.padded_problem(rho, rho)]
    u, v = k[2].clone(), k[2].clone()
    lmg.solve(*k, u, 20.0, 20.0, method=getattr(lmg, method), eps=1e-10)
    O.set_option("heat_wait_ms", 0)
    try:
        with pytest.raises(_lib.OpsError, match="wait between thread blocks expired"):
            lmg.solve(*k, v, 20.0, 20.0, method=getattr(lmg, method), eps=1e-10)
    finally:
        O.set_option("heat_wait_ms", 2000)
    assert torch.equal(v, k[2])
    lmg.solve(*k, v, 20.0, 20.0, method=getattr(lmg, method), eps=1e-10)
    assert torch.equal(u, v)
    with pytest.raises(_lib.OpsError):
        O.set_option("heat_wait_ms", -1)
