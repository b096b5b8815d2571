"""Performance cases of OPS-B200: the work its users have it do, through the
public entry points.

Seven families, each the shape of one of the framework's configurations:

  laplace   Jacobi sweeps queued with ops_par_loop, the residual read back
            after every sweep (the loop condition of the tutorial app)
  clover2d  whole CloverLeaf 2D runs (apps.cloverleaf), a summary each step
  clover3d  whole CloverLeaf 3D runs (apps.cloverleaf3d)
  adi       batched tridiagonal sweeps along x, y and z (trid_batch on device
            pointers, or ops_tridMultiDimBatch on dats)
  heat2d    implicit heat solves to 1e-10 (lmg.solve: FP64 PCG, mixed
            precision, multigrid-preconditioned flexible CG)
  heat3d    the 7-point solve (lmg.solve3d)
  net       the learned preconditioner: its application and a training step
"""
import numpy as np
import torch

from ops_b200 import apps, lmg, seeded
from ops_b200 import ops as O

F64 = torch.float64


def listed():
    return [
        # the smallest call: a tutorial-size grid, a few sweeps; launches and read-backs are all there is
        dict(name="laplace_96x64", family="laplace", nx=96, ny=64, iters=10),
        # the 4096^2 Jacobi configuration, twenty sweeps of its thousand
        dict(name="laplace_4096", family="laplace", nx=4096, ny=4096, iters=20),
        # a hydro run on a small odd-shaped mesh: about forty short loops a step
        dict(name="clover2d_250x187", family="clover2d", nx=250, ny=187, steps=10),
        # the 3840^2 hydro configuration, ten steps of its two hundred
        dict(name="clover2d_3840", family="clover2d", nx=3840, ny=3840, steps=10),
        # the 256^3 hydro run, four steps
        dict(name="clover3d_256", family="clover3d", nx=256, ny=256, nz=256, steps=4),
        # one ADI step of the single-block configuration, FP64
        dict(name="adi_cube_256_f64", family="adi", lo=256, hi=256, blocks=1, dtype="f64", api="batch", shapes=3),
        # the uneven multi-block configuration, FP32
        dict(name="adi_blocks64_f32", family="adi", lo=32, hi=192, blocks=64, dtype="f32", api="batch", shapes=3),
        # a training-size solve: one small grid, hundreds of short iterations
        dict(name="heat2d_pcg_128", family="heat2d", nx=128, ny=128, rx=400.0, method="pcg_true"),
        # the plain FP64 solve of the 4096^2 heat configuration
        dict(name="heat2d_pcg_4096", family="heat2d", nx=4096, ny=4096, rx=671.0, method="pcg_true"),
        # the same problem with the native multigrid preconditioner
        dict(name="heat2d_mg_4096", family="heat2d", nx=4096, ny=4096, rx=671.0, method="mg"),
        # the 7-point solve in mixed precision
        dict(name="heat3d_mixed_192", family="heat3d", nx=192, ny=192, nz=192, rx=100.0, method="mixed"),
        # one step of the training recipe: a batch of sixteen 64^2 pairs, forward, backward and Adam
        dict(name="net_train_16x64", family="net", n=16, ny=64, nx=64, op="train"),
    ]


def _log(rng, lo, hi):
    """A whole number, log-uniform in [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    family = rng.choice(["laplace", "clover2d", "clover3d", "adi", "adi", "heat2d", "heat2d", "heat3d", "net", "net"])
    if family == "laplace":
        return dict(family=family, nx=_log(rng, 48, 4096), ny=_log(rng, 48, 4096), iters=rng.randint(5, 20))
    if family == "clover2d":
        n = _log(rng, 48, 3072)
        return dict(family=family, nx=n, ny=max(32, int(n * rng.uniform(0.6, 1.25))), steps=rng.randint(4, 10))
    if family == "clover3d":
        n = _log(rng, 24, 224)
        return dict(family=family, nx=n, ny=max(16, int(n * rng.uniform(0.7, 1.2))),
                    nz=max(16, int(n * rng.uniform(0.7, 1.2))), steps=rng.randint(2, 4))
    if family == "adi":
        dtype = rng.choice(["f64", "f32"])
        if rng.random() < 0.5:
            hi = _log(rng, 48, 256)
            return dict(family=family, lo=rng.randint(16, 40), hi=hi, blocks=rng.randint(2, 64), dtype=dtype,
                        api="batch", shapes=rng.randint(0, 10 ** 6))
        hi = _log(rng, 16, 288)
        return dict(family=family, lo=max(8, int(hi * rng.uniform(0.6, 1.0))), hi=hi, blocks=1, dtype=dtype,
                    api=rng.choice(["batch", "dats"]), shapes=rng.randint(0, 10 ** 6))
    if family == "heat2d":
        method = rng.choice(["pcg_true", "pcg", "mixed", "mg"])
        n = _log(rng, 48, 4096 if method == "mg" else 2560)
        return dict(family=family, nx=n, ny=max(32, int(n * rng.uniform(0.7, 1.2))), rx=float(rng.randint(50, 600)),
                    method=method)
    if family == "heat3d":
        n = _log(rng, 16, 224)
        return dict(family=family, nx=n, ny=max(12, int(n * rng.uniform(0.7, 1.2))),
                    nz=max(12, int(n * rng.uniform(0.7, 1.2))), rx=float(rng.randint(20, 150)),
                    method=rng.choice(["pcg_true", "mixed"]))
    # the network takes grids of multiples of 8
    if rng.random() < 0.5:
        return dict(family=family, n=rng.randint(4, 24), ny=8 * rng.randint(4, 16), nx=8 * rng.randint(4, 16),
                    op="train")
    n = _log(rng, 64, 2048)
    return dict(family=family, n=1, ny=max(8, n // 8 * 8), nx=max(8, int(n * rng.uniform(0.7, 1.2)) // 8 * 8),
                op="apply")


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _init():
    global _ready
    if not _ready:
        O.ops_init(0, 0)
        _ready = True


_ready = False


class _Strided:
    """A device pointer of the runtime as an array for torch."""

    def __init__(self, ptr, shape, strides, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, strides=strides, typestr=typestr,
                                             version=3)


def _view(dat, shape):
    """The cells of a dat (numpy order, halo-free) where they lie on the GPU."""
    ptr, st = O.ops_dat_get_raw_pointer(dat, O.OPS_DEVICE)
    O.ops_dat_release_raw_data(dat, O.OPS_READ)
    es = 8 if dat.type == "double" else 4
    strides = [es, es * st[0], es * st[0] * st[1]][:len(shape)][::-1]
    return torch.as_tensor(_Strided(ptr, tuple(shape), tuple(strides), "<f%d" % es), device="cuda")


def _laplace_field(case, seed):
    """Boundary ring uniform in [0, 1), interior zero."""
    rng = np.random.default_rng(seed)
    f = np.zeros((case["ny"] + 2, case["nx"] + 2))
    f[0], f[-1] = rng.random(f.shape[1]), rng.random(f.shape[1])
    f[:, 0], f[:, -1] = rng.random(f.shape[0]), rng.random(f.shape[0])
    return f


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _adi_shapes(case):
    """Block shapes (numpy order z, y, x), edges log-uniform in [lo, hi]."""
    u = seeded.u01(case["shapes"], np.arange(3 * case["blocks"], dtype=np.uint64)).reshape(-1, 3)
    return [tuple(int(round(case["lo"] * (case["hi"] / case["lo"]) ** v)) for v in row) for row in u]


def _adi_data(case, seed):
    """Per block: a = c = -lam, b = 1 + 2 lam with lam ~ U[0.1, 1] per line,
    right-hand sides N(0, 1) and a start field u; every array a flat tensor
    over all blocks."""
    dt = F64 if case["dtype"] == "f64" else torch.float32
    g = _gen(seed)
    shapes = _adi_shapes(case)
    sizes = [z * y * x for z, y, x in shapes]
    total = sum(sizes)
    lam = torch.empty(total, dtype=dt, device="cuda")
    at = 0
    for (z, y, x), n in zip(shapes, sizes):
        line = torch.rand((z, y, 1), dtype=F64, device="cuda", generator=g) * 0.9 + 0.1
        lam[at:at + n] = line.expand(z, y, x).reshape(-1).to(dt)
        at += n
    rhs = torch.randn(total, dtype=dt, device="cuda", generator=g)
    u = torch.randn(total, dtype=dt, device="cuda", generator=g)
    return shapes, sizes, -lam, 1 + 2 * lam, -lam, rhs, u


def _density2d(ny, nx, seed):
    """Density and energy of the seeded heat problem: 16 rectangles, density
    log-uniform in [0.1, 100], over a background of 1."""
    st = seeded.tea_config4_states(nx, ny, int(seed))
    rho = torch.full((ny, nx), st[0]["density"], dtype=F64, device="cuda")
    en = torch.full((ny, nx), st[0]["energy"], dtype=F64, device="cuda")
    for s in st[1:]:
        x0, x1 = round(s["xmin"] * nx / 10), round(s["xmax"] * nx / 10)
        y0, y1 = round(s["ymin"] * ny / 10), round(s["ymax"] * ny / 10)
        rho[y0:y1, x0:x1] = s["density"]
        en[y0:y1, x0:x1] = s["energy"]
    return rho, en


def _heat2d_data(ny, nx, seed):
    rho, en = _density2d(ny, nx, seed)
    Kx, Ky, u0 = (torch.zeros((ny + 2, nx + 2), dtype=F64, device="cuda") for _ in range(3))
    Kx[1:-1, 2:-1] = (rho[:, :-1] + rho[:, 1:]) / (2.0 * rho[:, :-1] * rho[:, 1:])
    Ky[2:-1, 1:-1] = (rho[:-1] + rho[1:]) / (2.0 * rho[:-1] * rho[1:])
    u0[1:-1, 1:-1] = en * rho
    return Kx, Ky, u0


def _heat3d_data(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    rng = np.random.default_rng(seed)
    rho = torch.ones((nz, ny, nx), dtype=F64, device="cuda")
    for _ in range(16):
        box = []
        for n in (nz, ny, nx):
            lo = int(rng.integers(0, n - 1))
            box.append(slice(lo, min(n, lo + int(rng.integers(max(1, n // 16), max(2, n // 3))))))
        rho[tuple(box)] = float(np.exp(rng.uniform(np.log(0.1), np.log(100.0))))
    en = torch.rand((nz, ny, nx), dtype=F64, device="cuda", generator=_gen(seed))
    Kx, Ky, Kz, u0 = (torch.zeros((nz + 2, ny + 2, nx + 2), dtype=F64, device="cuda") for _ in range(4))
    c = slice(1, -1)
    w = rho
    Kx[c, c, 2:-1] = (w[:, :, :-1] + w[:, :, 1:]) / (2.0 * w[:, :, :-1] * w[:, :, 1:])
    Ky[c, 2:-1, c] = (w[:, :-1] + w[:, 1:]) / (2.0 * w[:, :-1] * w[:, 1:])
    Kz[2:-1, c, c] = (w[:-1] + w[1:]) / (2.0 * w[:-1] * w[1:])
    u0[c, c, c] = en * rho
    return Kx, Ky, Kz, u0


def _apply2d(Kx, Ky, u, rx):
    """A u on the interior of padded arrays (any leading batch dimensions)."""
    c = (Ellipsis, slice(1, -1), slice(1, -1))
    e, w = (Ellipsis, slice(1, -1), slice(2, None)), (Ellipsis, slice(1, -1), slice(None, -2))
    n, s = (Ellipsis, slice(2, None), slice(1, -1)), (Ellipsis, slice(None, -2), slice(1, -1))
    out = torch.zeros_like(u)
    out[c] = ((1.0 + rx * (Ky[n] + Ky[c] + Kx[e] + Kx[c])) * u[c] - rx * (Ky[n] * u[n] + Ky[c] * u[s])
              - rx * (Kx[e] * u[e] + Kx[c] * u[w]))
    return out


def _net_data(case, seed):
    """Pairs (r, e) with r = A e on seeded coefficient fields, rx = 1 with the
    timestep folded into the coefficients (as the training recipe makes them)."""
    n, ny, nx = case["n"], case["ny"], case["nx"]
    g = _gen(seed)
    Kx, Ky, e = (torch.zeros((n, ny + 2, nx + 2), dtype=F64, device="cuda") for _ in range(3))
    for i in range(n):
        Kx[i], Ky[i], _ = _heat2d_data(ny, nx, seed * 64 + i)
    scale = 100.0 * 10.0 ** torch.rand((n, 1, 1), dtype=F64, device="cuda", generator=g)
    Kx *= scale
    Ky *= scale
    e[:, 1:-1, 1:-1] = torch.randn((n, ny, nx), dtype=F64, device="cuda", generator=g)
    return Kx, Ky, e, _apply2d(Kx, Ky, e, 1.0)


def _net_params(seed):
    """He-normal convolutions with small biases and an output layer that, as
    in a network under training, is no longer zero."""
    rng = np.random.default_rng(seed)
    p = []
    for cin, cout in _LAYERS:
        p += [(2.0 / (9.0 * cin)) ** 0.5 * rng.standard_normal(9 * cin * cout), 0.05 * rng.standard_normal(cout)]
    p.append(0.1 * rng.standard_normal(17))
    return np.concatenate(p).astype(np.float32)


_LAYERS = [(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 64), (64, 64), (64, 32), (32, 16), (16, 16)]


class _Network:
    """A network handle that is given back with the state that holds it."""

    def __init__(self, seed):
        self.net = lmg.Net(5)
        self.net.set_params(_net_params(seed))

    def __del__(self):
        try:
            self.net.close()
        except Exception:
            pass


_METHOD = dict(pcg=lmg.PCG, pcg_true=lmg.PCG_TRUE, mixed=lmg.MIXED, mg=lmg.FCG_MG)


def prepare(case, seed):
    _init()
    f = case["family"]
    st = dict(case=case)
    if f == "laplace":
        init = _laplace_field(case, seed)
        st["grid"] = grid = O.ops_decl_block(2, "grid")
        size, base, m, p = [case["nx"], case["ny"]], [0, 0], [-1, -1], [1, 1]
        st["A"] = O.ops_decl_dat(grid, 1, size, base, m, p, init, "double", "A")
        st["Anew"] = O.ops_decl_dat(grid, 1, size, base, m, p, init, "double", "Anew")
        st["S0"] = O.ops_decl_stencil(2, 1, [0, 0], "0,0")
        st["S5"] = O.ops_decl_stencil(2, 5, [0, 0, 1, 0, -1, 0, 0, 1, 0, -1], "5pt")
        st["err"] = O.ops_decl_reduction_handle(8, "double", "error")
    elif f == "clover2d":
        st["deck"] = apps.clover_deck(x_cells=case["nx"], y_cells=case["ny"], xmax=10.0, ymax=10.0,
                                      initial_timestep=0.04, timestep_rise=1.5, max_timestep=0.04,
                                      end_step=case["steps"], summary_frequency=1,
                                      states=seeded.clover_config2_states(case["nx"], case["ny"], int(seed)))
    elif f == "clover3d":
        dims = (case["nx"], case["ny"], case["nz"])
        st["deck"] = apps.clover3d_deck(x_cells=dims[0], y_cells=dims[1], z_cells=dims[2], xmax=10.0, ymax=10.0,
                                        zmax=10.0, initial_timestep=0.04, timestep_rise=1.5, max_timestep=0.04,
                                        end_step=case["steps"], summary_frequency=1,
                                        states=seeded.clover3d_states(*dims, int(seed)))
    elif f == "adi":
        shapes, sizes, a, b, c, rhs, u = _adi_data(case, seed)
        if case["api"] == "dats":
            (z, y, x), ty = shapes[0], "double" if case["dtype"] == "f64" else "float"
            blk = O.ops_decl_block(3, "adi")
            for name, t in (("a", a), ("b", b), ("c", c), ("d", rhs), ("u", u)):
                st[name] = O.ops_decl_dat(blk, 1, [x, y, z], [0, 0, 0], [0, 0, 0], [0, 0, 0],
                                          t.reshape(z, y, x).cpu().numpy(), ty, name)
            st["range"], st["shape"] = [0, x, 0, y, 0, z], (z, y, x)
            return st
        d = torch.empty_like(rhs)
        st.update(a=a, b=b, c=c, d=d, u=u, rhs=rhs, es=a.element_size())
        st["plain"], st["inc"] = [], []
        at = 0
        for shp, n in zip(shapes, sizes):
            one = {k: t.data_ptr() + at * st["es"] for k, t in (("a", a), ("b", b), ("c", c), ("d", d), ("u", u))}
            one.update(dims=list(shp[::-1]), pads=list(shp[::-1]))
            st["inc"].append(one)
            st["plain"].append(dict(one, u=None))
            at += n
    elif f == "heat2d":
        st["Kx"], st["Ky"], st["u0"] = _heat2d_data(case["ny"], case["nx"], seed)
        st["u"] = torch.empty_like(st["u0"])
    elif f == "heat3d":
        st["Kx"], st["Ky"], st["Kz"], st["u0"] = _heat3d_data(case, seed)
        st["u"] = torch.empty_like(st["u0"])
    else:
        st["Kx"], st["Ky"], st["e"], st["r"] = _net_data(case, seed)
        st["out"] = torch.zeros_like(st["r"])
        st["network"] = _Network(seed)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    f = case["family"]
    if f == "laplace":
        grid, A, Anew, S0, S5, err = (state[k] for k in ("grid", "A", "Anew", "S0", "S5", "err"))
        rng = [0, case["nx"], 0, case["ny"]]
        errors = []
        for _ in range(case["iters"]):
            O.ops_par_loop("laplace2d/apply_stencil", "apply_stencil", grid, 2, rng,
                           O.ops_arg_dat(A, 1, S5, "double", O.OPS_READ),
                           O.ops_arg_dat(Anew, 1, S0, "double", O.OPS_WRITE),
                           O.ops_arg_reduce(err, 1, "double", O.OPS_MAX))
            errors.append(float(O.ops_reduction_result(err)))
            O.ops_par_loop("laplace2d/copy", "copy", grid, 2, rng,
                           O.ops_arg_dat(A, 1, S0, "double", O.OPS_WRITE),
                           O.ops_arg_dat(Anew, 1, S0, "double", O.OPS_READ))
        return dict(field=_view(A, (case["ny"], case["nx"])), errors=np.array(errors))
    if f == "clover2d":
        return apps.cloverleaf(state["deck"])[0]
    if f == "clover3d":
        return apps.cloverleaf3d(state["deck"])[0]
    if f == "adi":
        if case["api"] == "dats":
            a, b, c, d, u = (state[k] for k in "abcdu")
            O.ops_tridMultiDimBatch(3, 0, state["range"], a, b, c, d)
            O.ops_tridMultiDimBatch(3, 1, state["range"], a, b, c, d)
            O.ops_tridMultiDimBatch_Inc(3, 2, state["range"], a, b, c, d, u)
            return dict(d=_view(d, state["shape"]), u=_view(u, state["shape"]))
        state["d"].copy_(state["rhs"])  # this step's right-hand side
        O.trid_batch(state["es"], 0, state["plain"])
        O.trid_batch(state["es"], 1, state["plain"])
        O.trid_batch(state["es"], 2, state["inc"])
        return dict(d=state["d"], u=state["u"])
    if f == "heat2d":
        state["u"].copy_(state["u0"])
        lmg.solve(state["Kx"], state["Ky"], state["u0"], state["u"], case["rx"], case["rx"],
                  method=_METHOD[case["method"]], eps=1e-10)
        return state["u"]
    if f == "heat3d":
        state["u"].copy_(state["u0"])
        lmg.solve3d(state["Kx"], state["Ky"], state["Kz"], state["u0"], state["u"], case["rx"], case["rx"],
                    case["rx"], method=_METHOD[case["method"]], eps=1e-10)
        return state["u"]
    net = state["network"].net
    if case["op"] == "apply":
        net.apply(state["r"], state["Kx"], state["Ky"], 1.0, 1.0, state["out"])
        return state["out"]
    # the late phase of the training recipe: its rate times 0.1
    loss = net.train_step(state["r"], state["Kx"], state["Ky"], state["e"], 1.0, 1.0, 2e-4)
    return dict(loss=loss, grads=net.grads())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    f = case["family"]
    if f == "laplace":  # every sweep reads and writes the field: its residual decides about the next
        cells = case["nx"] * case["ny"] * case["iters"]
        return dict(bytes=16.0 * cells, flops=6.0 * cells)
    if f == "clover2d":
        # a step has one global barrier, the CFL minimum: before it density, energy, two velocities, volume and two
        # areas in, pressure, viscosity and sound speed out; after it these ten in and the step's new density,
        # energy, velocities and volume and mass fluxes out
        cells = case["nx"] * case["ny"] * case["steps"]
        return dict(bytes=8.0 * (7 + 3 + 10 + 8) * cells, flops=700.0 * cells)
    if f == "clover3d":
        cells = case["nx"] * case["ny"] * case["nz"] * case["steps"]
        return dict(bytes=8.0 * (9 + 3 + 12 + 11) * cells, flops=1600.0 * cells)
    if f == "adi":  # three sweeps: a, b, c and the right-hand side in, the solution out; the last adds it to u
        n = sum(z * y * x for z, y, x in _adi_shapes(case))
        return dict(bytes=(8.0 if case["dtype"] == "f64" else 4.0) * (5 + 5 + 6) * n, flops=3 * 8.0 * n)
    if f == "heat2d":
        cells = case["nx"] * case["ny"]
        if case["method"] == "mg":  # about 15 iterations; w, u, r, p in FP64 and one V-cycle in FP32
            return dict(bytes=15.0 * 180 * cells, flops=15.0 * 150 * cells)
        # iterations grow with the square root of the condition number; each
        # reads the operator and updates p, w, r and u
        iters = 66.0 * case["rx"] ** 0.5 * min(1.0, (cells ** 0.5 / 1024) ** 0.35)
        return dict(bytes=iters * (36.0 if case["method"] == "mixed" else 72.0) * cells, flops=iters * 24 * cells)
    if f == "heat3d":
        cells = case["nx"] * case["ny"] * case["nz"]
        iters = 36.0 * case["rx"] ** 0.5
        return dict(bytes=iters * (40.0 if case["method"] == "mixed" else 80.0) * cells, flops=iters * 30 * cells)
    px = case["n"] * case["nx"] * case["ny"]
    # multiply-adds per fine pixel: a level's grid has a quarter of the cells of the one above
    level = [0, 1, 1, 2, 2, 3, 3, 2, 1, 0]
    macs = sum(9.0 * ci * co / 4 ** lv for (ci, co), lv in zip(_LAYERS, level))
    if case["op"] == "apply":  # r and the faces in, the result out, the skip tensors kept in between
        return dict(bytes=px * (3 * 8.0 + 8.0 + 2 * 32.0), flops=2.0 * macs * px)
    return dict(bytes=px * (4 * 8.0 + 4 * 32.0), flops=6.0 * macs * px)


# ---------------------------------------------------------------------------
# 64-bit results by plain torch
# ---------------------------------------------------------------------------
def _thomas(a, b, c, d, dim):
    """Tridiagonal solve along `dim` in 64 bits."""
    a, b, c, d = (t.to(F64).movedim(dim, 0) for t in (a, b, c, d))
    n = b.shape[0]
    cp, dp = [c[0] / b[0]], [d[0] / b[0]]
    for i in range(1, n):
        m = b[i] - a[i] * cp[-1]
        cp.append(c[i] / m)
        dp.append((d[i] - a[i] * dp[-1]) / m)
    x = [dp[-1]]
    for i in range(n - 2, -1, -1):
        x.append(dp[i] - cp[i] * x[-1])
    return torch.stack(x[::-1]).movedim(0, dim)


def _cg(apply, diag, b, u):
    """Jacobi-PCG to a residual of 1e-13 of the first."""
    r = b - apply(u)
    z = r / diag
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-13 * r.norm()
    for it in range(20000):
        w = apply(p)
        alpha = rz / (p * w).sum()
        u = u + alpha * p
        r -= alpha * w
        if it % 16 == 15 and bool(r.norm() < stop):
            break
        z = r / diag
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return u


def _conv(x, w, b):
    """3x3 convolution of NHWC images, w [9, cout, cin], then ReLU."""
    n, h, wd, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out = b.expand(n, h, wd, b.numel())
    for t in range(9):
        out = out + xp[:, t // 3:t // 3 + h, t % 3:t % 3 + wd] @ w[t].T
    return torch.relu(out)


def _network(params, r, Kx, Ky):
    """M(r) of the learned preconditioner in 64 bits; params a flat tensor."""
    layers, at = [], 0
    for cin, cout in _LAYERS:
        w = params[at:at + 9 * cin * cout].reshape(9, cout, cin)
        at += 9 * cin * cout
        layers.append((w, params[at:at + cout]))
        at += cout
    wout, bout = params[at:at + 16], params[at + 16]
    i = slice(1, -1)
    k = [Kx[:, i, i], Kx[:, i, 2:], Ky[:, i, i], Ky[:, 2:, i]]
    D = 1.0 + k[0] + k[1] + k[2] + k[3]
    ri = r[:, i, i]
    s = ri.square().mean((1, 2), keepdim=True).sqrt()
    x = torch.stack([ri / s] + [q / D for q in k], -1)
    x = torch.nn.functional.pad(x, (0, 11))
    n, h, w, _ = x.shape

    def pool(t):
        return t.reshape(t.shape[0], t.shape[1] // 2, 2, t.shape[2] // 2, 2, t.shape[3]).mean((2, 4))

    def up(t):
        return t.repeat_interleave(2, 1).repeat_interleave(2, 2)

    e0 = _conv(x, *layers[0])
    e1 = _conv(_conv(pool(e0), *layers[1]), *layers[2])
    e2 = _conv(_conv(pool(e1), *layers[3]), *layers[4])
    h3 = _conv(_conv(pool(e2), *layers[5]), *layers[6])
    h2 = _conv(up(h3) + e2, *layers[7])
    h1 = _conv(up(h2) + e1, *layers[8])
    h0 = _conv(up(h1) + e0, *layers[9])
    return ri / D + s * (h0 @ wout + bout)


def exact(case, seed):
    f = case["family"]
    if f == "laplace":
        A = torch.from_numpy(_laplace_field(case, seed)).cuda()
        errors = []
        for _ in range(case["iters"]):
            new = 0.25 * (A[1:-1, 2:] + A[1:-1, :-2] + A[2:, 1:-1] + A[:-2, 1:-1])
            errors.append(float((new - A[1:-1, 1:-1]).abs().max()))
            A[1:-1, 1:-1] = new
        return dict(field=A[1:-1, 1:-1].contiguous(), errors=np.array(errors))
    if f in ("clover2d", "clover3d"):
        return None
    if f == "adi":
        shapes, sizes, a, b, c, rhs, u = _adi_data(case, seed)
        d_out, u_out, at = [], [], 0
        for shp, n in zip(shapes, sizes):
            A, B, C, d, U = (t[at:at + n].reshape(shp) for t in (a, b, c, rhs, u))
            d = _thomas(A, B, C, _thomas(A, B, C, d, 2), 1)
            d_out.append(d.reshape(-1))
            u_out.append((U.to(F64) + _thomas(A, B, C, d, 0)).reshape(-1))
            at += n
        d_all, u_all = torch.cat(d_out), torch.cat(u_out)
        if case["api"] == "dats":
            return dict(d=d_all.reshape(shapes[0]), u=u_all.reshape(shapes[0]))
        return dict(d=d_all, u=u_all)
    if f == "heat2d":
        Kx, Ky, u0 = _heat2d_data(case["ny"], case["nx"], seed)
        rx = case["rx"]
        diag = torch.ones_like(u0)
        c = slice(1, -1)
        diag[c, c] = 1.0 + rx * (Ky[2:, c] + Ky[c, c] + Kx[c, 2:] + Kx[c, c])
        return _cg(lambda v: _apply2d(Kx, Ky, v, rx), diag, u0, u0.clone())
    if f == "heat3d":
        Kx, Ky, Kz, u0 = _heat3d_data(case, seed)
        rx, c = case["rx"], slice(1, -1)
        diag = torch.ones_like(u0)
        diag[c, c, c] = 1.0 + rx * (Kz[2:, c, c] + Kz[c, c, c] + Ky[c, 2:, c] + Ky[c, c, c] + Kx[c, c, 2:] + Kx[c, c, c])

        def op(v):
            out = torch.zeros_like(v)
            out[c, c, c] = (diag[c, c, c] * v[c, c, c]
                            - rx * (Kz[2:, c, c] * v[2:, c, c] + Kz[c, c, c] * v[:-2, c, c])
                            - rx * (Ky[c, 2:, c] * v[c, 2:, c] + Ky[c, c, c] * v[c, :-2, c])
                            - rx * (Kx[c, c, 2:] * v[c, c, 2:] + Kx[c, c, c] * v[c, c, :-2]))
            return out

        return _cg(op, diag, u0, u0.clone())
    Kx, Ky, e, r = _net_data(case, seed)
    params = torch.from_numpy(_net_params(seed).astype(np.float64)).cuda()
    if case["op"] == "apply":
        out = torch.zeros_like(r)
        out[:, 1:-1, 1:-1] = _network(params, r, Kx, Ky)
        return out
    params.requires_grad_(True)
    d = torch.zeros_like(r)
    d[:, 1:-1, 1:-1] = _network(params, r, Kx, Ky) - e[:, 1:-1, 1:-1]
    c = (slice(None), slice(1, -1), slice(1, -1))
    num = (d * _apply2d(Kx, Ky, d, 1.0))[c].sum((1, 2))
    den = (e * r)[c].sum((1, 2))
    loss = (num / den).mean()
    loss.backward()
    return dict(loss=float(loss), grads=params.grad.cpu().numpy())
