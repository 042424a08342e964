"""PDE structs of other shapes than the library's own compile against the kernels
(CPU) and give right results (GPU): a linear PDE without parameters, one with
unequal numbers of gradient components per direction, and one with more than 16
values per node in the Riemann solver. An order without transfer tables does not
compile (it would read another order's).

Bounds: the same sums in another order, 1e-12 of the largest value (the derivative
tables are read from the same generator)."""
import ctypes
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "exahype_b200", "csrc")
NVCC = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else shutil.which("nvcc")
RTOL = 1e-12


def compile_ext(out, *flags):
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                           "--expt-relaxed-constexpr", "-I", CSRC, *flags, os.path.join(HERE, "pde_extension.cu"),
                           "-o", str(out)])


@pytest.mark.skipif(not NVCC, reason="needs nvcc")
def test_other_pde_shapes_compile(tmp_path):
    compile_ext(tmp_path / "ext.o", "-c")


@pytest.mark.skipif(not NVCC, reason="needs nvcc")
def test_orders_without_tables_do_not_compile(tmp_path):
    src = tmp_path / "t.cu"
    src.write_text('#include "amr.cuh"\n'
                   "template __global__ void exa::plot_vertex_kernel<2, ORDER, 5>(const double*, double*, int);\n")
    run = lambda order: subprocess.run(  # noqa: E731
        [NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
         "-DORDER=%d" % order, "-c", str(src), "-o", str(tmp_path / "t.o")], capture_output=True, text=True)
    assert run(5).returncode == 0
    r = run(6)
    assert r.returncode != 0 and "no transfer tables" in r.stderr


@pytest.mark.skipif(not NVCC, reason="needs nvcc")
def test_tensor_memory_predictor_refuses_idle_threads(tmp_path):
    """order 2 in 2D: 126 nodes in a block of 128 threads and more lines than nodes"""
    src = tmp_path / "t.cu"
    src.write_text('#include "aderdg.cuh"\n#include "predictor_tmem.cuh"\n'
                   "static_assert(exa::TmemCfg<2, ORDER, exa::EulerPDE>::THREADS == 128);\n")
    run = lambda order: subprocess.run(  # noqa: E731
        [NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
         "-DORDER=%d" % order, "-c", str(src), "-o", str(tmp_path / "t.o")], capture_output=True, text=True)
    assert run(3).returncode == 0
    r = run(2)
    assert r.returncode != 0 and "a node for every thread" in r.stderr


@pytest.fixture(scope="module")
def ext(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    out = tmp_path_factory.mktemp("ext") / "libext.so"
    compile_ext(out, "-shared", "-Xcompiler", "-fPIC")
    torch.cuda.init()
    lib = ctypes.CDLL(str(out))
    assert lib.ext_tables() == 0
    return lib


def tables(order):
    sys.path.insert(0, CSRC)
    try:
        import gen_tables
    finally:
        sys.path.pop(0)
    t, b = gen_tables.build(order), order + 1
    return dict(w=np.array(t["weights"]), FL=np.array(t["FLCoeff"]), FR=np.array(t["FRCoeff"]),
                D=np.array(t["dudx"]).reshape(b, b))


def rel(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


def predict(lib, which, luh, nv, F, dt, dx):
    import torch
    n, P, nd = luh.shape
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
    qb, fb, du = z(n, 2 * len(dx), F, nd), z(n, 2 * len(dx), F, nv), z(n, P, nv)
    a, t = torch.as_tensor(luh).cuda(), torch.tensor([dt], dtype=torch.float64, device="cuda")
    ptr = [ctypes.c_void_p(x.data_ptr()) for x in (a, qb, fb, du, t)]
    torch.cuda.synchronize()
    assert lib.ext_predictor(which, *ptr, (ctypes.c_double * 3)(*(list(dx) + [0.0] * (3 - len(dx)))), n) == 0
    torch.cuda.synchronize()
    return qb.cpu().numpy(), fb.cpu().numpy(), du.cpu().numpy()


def acoustic_product(d, G):
    B = np.zeros_like(G)
    B[..., 0], B[..., 1 + d] = 2.0 * G[..., 1 + d], 2.0 * G[..., 0]
    return B


@pytest.mark.gpu
@pytest.mark.parametrize("which,dim,order,n", [(0, 2, 3, 13), (1, 3, 3, 7), (5, 3, 5, 3)])
def test_linear_pde_without_parameters(ext, which, dim, order, n):
    rng = np.random.default_rng(which)
    T, b, dx, dt = tables(order), order + 1, [0.05, 0.04, 0.045][:dim], 1e-3
    luh = rng.normal(size=(n, b ** dim, 4))
    along = lambda a, d: np.moveaxis(np.tensordot(a, T["D"], axes=([dim - d], [1])), -1, dim - d)  # noqa: E731
    lev = luh.reshape([n] + [b] * dim + [4])
    qh, F, fac = lev.copy(), [0.0] * dim, 1.0
    for i in range(b):
        B = [acoustic_product(d, along(lev, d) / dx[d]) for d in range(dim)]
        for d in range(dim):
            F[d] = F[d] + fac * B[d]
        lev = -sum(B)
        fac = fac * dt / (i + 2)
        if i + 1 < b:
            qh = qh + fac * lev
    trace = lambda a, d, side: np.tensordot(a, T[side], axes=([dim - d], [0])).reshape(n, -1, 4)  # noqa: E731
    qb = np.stack([trace(qh, d, s) for d in range(dim) for s in ("FL", "FR")], axis=1)
    fb = np.stack([trace(F[d], d, s) for d in range(dim) for s in ("FL", "FR")], axis=1)
    w = T["w"]
    W = w[:, None] * w[None, :] if dim == 2 else w[:, None, None] * w[None, :, None] * w[None, None, :]
    du = -(W[None, ..., None] * sum(F)).reshape(n, -1, 4)
    for got, want in zip(predict(ext, which, luh, 4, b ** (dim - 1), dt, dx), (qb, fb, du)):
        assert rel(got, want) < RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("which,dim,order,n", [(2, 2, 5, 11), (3, 3, 3, 9), (4, 3, 5, 5)])
def test_uneven_components_equal_even_ones(ext, which, dim, order, n):
    """the elastic PDE with components it does not need, as many as it likes per direction"""
    import torch

    import exahype_b200 as eb
    rng = np.random.default_rng(which)
    b, dx, dt = order + 1, [0.05, 0.04, 0.045][:dim], 1e-3
    luh = rng.normal(size=(n, b ** dim, 12))
    luh[..., 9:] = 1.0 + rng.random((n, b ** dim, 3))
    got = predict(ext, which, luh, 9, b ** (dim - 1), dt, dx)
    s = eb.Solver(dim, order, eb.PDE_ELASTIC)
    out = [torch.zeros(g.shape, dtype=torch.float64, device="cuda") for g in got]
    t = torch.tensor([dt], dtype=torch.float64, device="cuda")
    s.space_time_predictor_linear(torch.as_tensor(luh).cuda(), *out, t, dx, n)
    torch.cuda.synchronize()
    for g, o in zip(got, out):
        assert rel(g, o.cpu().numpy()) < RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["acoustic", "wide"])
def test_riemann_solvers(ext, kind):
    import torch
    rng = np.random.default_rng(5)
    nd, nv = (4, 4) if kind == "acoustic" else (19, 18)
    n, F, w = 9, 16, tables(3)["w"]
    q, f = rng.normal(size=(n, 6, F, nd)), rng.normal(size=(n, 6, F, nv))
    l, d = np.arange(3 * n) // 3, np.arange(3 * n) % 3
    r = (l + 1) % n
    dev = [torch.as_tensor(a).cuda() for a in (q, f)] + [torch.as_tensor(a.astype(np.int32)).cuda() for a in (l, r, d)]
    torch.cuda.synchronize()
    call = ext.ext_riemann_linear if kind == "acoustic" else ext.ext_riemann_wide
    assert call(*[ctypes.c_void_p(a.data_ptr()) for a in dev], 3 * n) == 0
    torch.cuda.synchronize()
    wf = (w[:, None] * w[None, :]).reshape(-1)
    want = f.copy()
    for i in range(3 * n):
        L, R = (l[i], 2 * d[i] + 1), (r[i], 2 * d[i])
        dq = (q[R] - q[L])[:, :nv]
        if kind == "acoustic":
            B = acoustic_product(d[i], 0.5 * dq)
            want[L], want[R] = B - 2.0 * 0.5 * dq, B + 2.0 * 0.5 * dq
        else:
            av = [(wf[:, None] * q[s]).sum(0) for s in (L, R)]
            smax = max(np.max(np.abs((np.arange(18) - 9) * 0.1 * a[:18] * a[18] * (1 + d[i]))) for a in av)
            want[L] = want[R] = 0.5 * (f[L] + f[R]) - 0.5 * smax * dq
    assert rel(dev[1].cpu().numpy(), want) < RTOL
