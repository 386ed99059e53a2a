"""The line kernels (nkb_line_kernel.cuh) against the shape-generic kernels:
every operator on every shape, at the smallest and largest orders, point counts
whose shared-memory rows are rotated (4 and 8) and not, over-integration,
straight-sided and curved geometry; collections of one element per CTA, of several,
and of full CTAs with the last one partly filled."""
import numpy as np
import pytest

import nektar_b200 as nb
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

OPS = ("bwdtrans", "iproduct", "physderiv", "iproduct_deriv", "helmholtz", "linear_adr")
# two summation orders of the same sums: a few hundred roundings of 1.1e-16 (6e-8)
# that add up as a random walk, times the operators' cancellation (about 10)
TOL = {"fp64": 1e-13, "fp32": 5e-6}
# (modes, points in the first direction)
SIZES = [(2, 3), (3, 4), (4, 5), (6, 7), (7, 8), (8, 9), (9, 10), (11, 12), (2, 4), (3, 6), (4, 8),
         (6, 8), (7, 11), (10, 12)]


def _apply(op, x, dtype):
    import torch
    nout = 3 if op.optype == nb.PHYSDERIV else 1
    xd = torch.tensor(x, dtype=dtype, device="cuda")
    out = torch.full((nout, op.out_size), float("nan"), dtype=dtype, device="cuda")
    op.apply_device(xd.data_ptr(), *[o.data_ptr() for o in out],
                    stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.double().cpu().numpy().ravel()


def _operator(name, mesh, precision, rng):
    op = nb.Operator(name, mesh, precision=precision)
    if name == "helmholtz":
        op.set_factors(0.7, nb.DIFF_CONST, [1.5, 0.2, 0.8, -0.1, 0.3, 1.1])
    if name == "linear_adr":
        op.set_factors(0.7)
        op.set_varcoeffs(*rng.uniform(-1, 1, (3, mesh.nelmt * mesh.nt)))
    return op


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("amp", [0.05, 0.0])
@pytest.mark.parametrize("nm,nq", SIZES)
@pytest.mark.parametrize("shape", ["hex", "prism", "tet"])
def test_line_and_generic_kernels_agree(monkeypatch, shape, nm, nq, amp, precision):
    import torch
    dtype = torch.float64 if precision == "fp64" else torch.float32
    for n in ([1, 3] if nm < 9 else [1]):
        m = nb.BoxMesh(shape, n, nm, nq, amp=amp)
        for name in OPS:
            line = _operator(name, m, precision, np.random.default_rng(nm))
            monkeypatch.setenv("NKB_KERNEL", "generic")
            generic = _operator(name, m, precision, np.random.default_rng(nm))
            monkeypatch.delenv("NKB_KERNEL")
            assert generic.kernel() == "k_generic"
            x = np.random.default_rng(nq).uniform(-1, 1, line.in_size)
            y, z = _apply(line, x, dtype), _apply(generic, x, dtype)
            assert rel_l2(y, z) < TOL[precision], (name, n, line.kernel())


def _full_cta_elements(shape, nq):
    """A count that fills every CTA, whatever the elements per CTA: more than all
    threads of the device at one line of points each."""
    import torch
    lines = nq * (nq if shape != "tet" else nq - 1)
    return torch.cuda.get_device_properties(0).multi_processor_count * 2048 // lines + 1


def _random_operator(name, shape, nm, nq, nelmt, curved, precision):
    """Elements whose factors vary from one to the next (and from point to point)."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nelmt)
    T, q = nb.shape_tables(shape, nm, nq)
    nt = q[0] * q[1] * q[2]
    n = nelmt * nt if curved else nelmt
    rand = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64, device="cuda") * 2 - 1
    jac, df = 1 + 0.3 * rand(n), 0.25 * rand(9, n)
    df[0::4] += 1
    op = nb.Operator(name, shape=shape, nm=nm, nq=q, nelmt=nelmt, T=T, jac=jac, df=df,
                     deformed=curved, precision=precision)
    if name in ("helmholtz", "linear_adr"):
        op.set_factors(0.7)
    if name == "linear_adr":
        vel = rand(3, nelmt * nt)
        op.set_varcoeffs(*[v.data_ptr() for v in vel])
    return op


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nm,nq", [(2, 3), (3, 4), (4, 5), (5, 6), (7, 8), (8, 9), (10, 11), (2, 4),
                                   (4, 8), (5, 9)])
@pytest.mark.parametrize("shape", ["hex", "prism", "tet"])
def test_full_and_partly_filled_ctas(monkeypatch, shape, nm, nq, precision):
    """Collections beyond one wave, where each CTA takes as many elements as it can:
    of two consecutive counts at least one leaves the last CTA partly filled. Below
    it, a collection of half that size, at a few elements per CTA."""
    import torch
    dtype = torch.float64 if precision == "fp64" else torch.float32
    full = _full_cta_elements(shape, nq)
    monkeypatch.setenv("NKB_GENERIC_TUNE", "0")
    for k, name in enumerate(OPS):
        for nelmt in (full + nq, full + nq + 1, full // 3):
            for curved in (True, False):
                if name == "bwdtrans" and not curved:
                    continue  # no geometry
                args = name, shape, nm, nq, nelmt, curved, precision
                line = _random_operator(*args)
                monkeypatch.setenv("NKB_KERNEL", "generic")
                generic = _random_operator(*args)
                monkeypatch.delenv("NKB_KERNEL")
                assert line.kernel().startswith("k_line") and generic.kernel() == "k_generic"
                x = torch.rand(line.in_size, dtype=dtype, device="cuda") * 2 - 1
                s = torch.cuda.current_stream().cuda_stream
                nout = 3 if name == "physderiv" else 1
                y, z = (torch.full((nout, op.out_size), float("nan"), dtype=dtype, device="cuda")
                        for op in (line, generic))
                for op, out in ((line, y), (generic, z)):
                    op.apply_device(x.data_ptr(), *[o.data_ptr() for o in out], stream=s)
                d, z = (y.double() - z.double()).view(nout, nelmt, -1), z.double().view(nout, nelmt, -1)
                # of every element by itself: the largest of 1e4 to 1e5 of them lies
                # within ten times the bound that holds for all together
                each = d.square().sum((0, 2)).sqrt() / z.square().sum((0, 2)).mean().sqrt()
                assert d.norm() < TOL[precision] * z.norm(), args
                assert each.max() < 10 * TOL[precision], args
                line.close(), generic.close()


@pytest.mark.parametrize("shape,nm,nq", [("hex", 3, 4), ("prism", 5, 6), ("tet", 4, 5), ("tet", 6, 9)])
def test_gathered_launches_of_full_ctas(monkeypatch, shape, nm, nq):
    """Three CG iterations of a block-diagonal system with signs and a permuted map,
    on full CTAs of the line and of the generic kernel."""
    nelmt = _full_cta_elements(shape, nq) + nq
    rng = np.random.default_rng(nq)
    nloc = nelmt * nb.ncoeffs(shape, nm)
    gmap, sign = rng.permutation(nloc).astype(np.int32), rng.choice([-1.0, 1.0], nloc)
    b, xs = rng.uniform(-1, 1, nloc), []
    for kernel in (None, "generic"):
        if kernel:
            monkeypatch.setenv("NKB_KERNEL", kernel)
        op = _random_operator("helmholtz", shape, nm, nq, nelmt, True, "fp64")
        S = nb.GlobalLinSys([op], gmap, nloc, 0, sign=sign)
        xs.append(S.solve(b, tol=1e-14, maxit=3, check_interval=3, raise_on_maxit=False)[0])
    # three iterations magnify the operators' TOL by a few times the ratio of
    # the largest to the smallest entry of the diagonal (about 1e2)
    assert np.abs(xs[0]).max() > 0 and rel_l2(*xs) < 1e2 * TOL["fp64"]


@pytest.mark.parametrize("shape", ["hex", "prism", "tet"])
@pytest.mark.parametrize("amp", [0.05, 0.0])
def test_line_kernel_diagonal_and_gather(monkeypatch, shape, amp):
    """The Helmholtz diagonal reads the line kernels' point order; a gathered
    launch with signs, through the CG of a block-diagonal system."""
    m = nb.BoxMesh(shape, 2, 5, 6, amp=amp)
    op = _operator("helmholtz", m, "fp64", None)
    nloc = m.nelmt * m.nc
    rng = np.random.default_rng(6)
    gmap = rng.permutation(nloc).astype(np.int32)
    sign = rng.choice([-1.0, 1.0], nloc)
    b = rng.uniform(-1, 1, nloc)
    monkeypatch.setenv("NKB_KERNEL", "generic")
    ref = _operator("helmholtz", m, "fp64", None)
    monkeypatch.delenv("NKB_KERNEL")
    assert rel_l2(op.helmholtz_diag(), ref.helmholtz_diag()) < 1e-13
    xs = [nb.GlobalLinSys([o], gmap, nloc, 0, sign=sign).solve(b, tol=1e-13)[0] for o in (op, ref)]
    assert rel_l2(*xs) < 1e-10


def test_line_kernel_three_input_fields_and_infinities():
    """IProductWRTDerivBase from three device arrays, and a value that is not
    finite, which must stay in its own element."""
    import torch
    m = nb.BoxMesh("tet", 2, 4, 5)
    op = nb.Operator("iproduct_deriv", m)
    f = torch.rand(3, m.nelmt * m.nt, dtype=torch.float64, device="cuda")
    f[1, 5 * m.nt + 3] = float("inf")
    y, z = (torch.empty(op.out_size, dtype=torch.float64, device="cuda") for _ in range(2))
    s = torch.cuda.current_stream().cuda_stream
    parts = [v.clone() for v in f]
    op.apply3_device(*[v.data_ptr() for v in parts], y.data_ptr(), stream=s)
    op.apply_device(f.data_ptr(), z.data_ptr(), stream=s)
    bad = ~torch.isfinite(y.view(m.nelmt, m.nc)).all(1)
    assert torch.equal(y.view(torch.int64), z.view(torch.int64))
    assert bad.nonzero().ravel().tolist() == [5]


def _pointwise(m, name, precision, scale=1.0):
    """The operator of m's straight-sided elements, and of the same elements given point
    by point as curved ones are; lengths scaled by `scale`."""
    rng = np.random.default_rng(m.nm)
    jac, df = m.jac * scale ** 3, m.df / scale
    vel = rng.uniform(-1, 1, (3, m.nelmt * m.nt))
    ops = []
    for deformed in (False, True):
        g = (np.repeat(jac, m.nt), np.repeat(df, m.nt, axis=1)) if deformed else (jac, df)
        op = nb.Operator(name, shape=m.shape, nm=m.nm, nq=m.nq, nelmt=m.nelmt, T=m.T, jac=g[0],
                         df=np.ascontiguousarray(g[1]), deformed=deformed, precision=precision)
        if name in ("helmholtz", "linear_adr"):
            op.set_factors(0.7)
        if name == "linear_adr":
            op.set_varcoeffs(*vel)
        ops.append(op)
    return ops


@pytest.mark.parametrize("name", ["helmholtz", "linear_adr"])
@pytest.mark.parametrize("nm,nq", [(2, 3), (4, 5), (5, 9), (8, 9), (11, 12)])
@pytest.mark.parametrize("shape", ["hex", "prism", "tet"])
def test_fp32_straight_sided_factors_are_rounded_once(shape, nm, nq, name):
    """FP32 operators on straight-sided elements use factors formed in FP64 and rounded
    once at each point: the bits of the same elements given point by point."""
    import torch
    m = nb.BoxMesh(shape, 2, nm, nq)
    assert not m.deformed
    straight, curved = _pointwise(m, name, "fp32")
    x = np.random.default_rng(nq).uniform(-1, 1, straight.in_size)
    assert np.array_equal(_apply(straight, x, torch.float32), _apply(curved, x, torch.float32))


@pytest.mark.parametrize("nm,nq", [(3, 4), (6, 7), (5, 9)])
@pytest.mark.parametrize("shape", ["hex", "prism", "tet"])
def test_fp32_straight_sided_metric_is_formed_in_fp64(shape, nm, nq):
    """IProductWRTDerivBase on elements whose Jacobian and weights (1e-45 and below)
    have no FP32 value, although their products with the derivative factors do."""
    import torch
    m = nb.BoxMesh(shape, 2, nm, nq)
    x = np.random.default_rng(nq).uniform(-1, 1, 3 * m.nelmt * m.nt)
    y = _apply(_pointwise(m, "iproduct_deriv", "fp32", 1e-14)[0], x, torch.float32)
    z = _apply(_pointwise(m, "iproduct_deriv", "fp64", 1e-14)[0], x, torch.float64)
    assert rel_l2(y, z) < TOL["fp32"]
