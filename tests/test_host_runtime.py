"""The library's host code on a CUDA runtime that runs nothing (cpp/fake_cudart.cpp):
faults that a GPU shows only now and then, or by ending the process."""
import os
import subprocess
import sys

import pytest

from tests.helpers import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp")
SHAPES = ("hex", "prism", "tet")
OPS = ("bwdtrans", "iproduct", "physderiv", "iproduct_deriv", "helmholtz", "linear_adr")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """The library's objects linked with the runtime's stand-in."""
    from nektar_b200 import build
    objs = [os.path.join(build.BUILD, s + ".o") for s in build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        pytest.skip("the objects of the build are not here")
    out = str(tmp_path_factory.mktemp("fake") / "libnekb200_fake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                           "-I" + inc, SRC] + objs + ["-ldl", "-o", out])
    return out


def run(lib, body, **env):
    """body in a process of its own, with nb, np, lib and mesh(shape, nm, n) defined."""
    head = ("import numpy as np\nimport nektar_b200 as nb\nfrom nektar_b200 import _capi as C\n"
            "C.LIB_PATH = %r\nlib = C.lib()\n"
            "SHAPES, OPS = %r, %r\n"
            "def mesh(shape, nm, n=1, amp=0.05):\n"
            "    return nb.BoxMesh(shape, n, nm, nm + 1, amp=amp)\n" % (lib, SHAPES, OPS))
    p = subprocess.run([sys.executable, "-c", head + body], cwd=ROOT, capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, **env))
    assert p.returncode == 0, (p.returncode, p.stderr[-3000:])


@pytest.mark.parametrize("env", [{}, {"NKB_HEX_VARIANT": "5"}, {"NKB_KERNEL": "generic"}])
def test_set_up_waits_for_its_copies(fake, env):
    """Operators, systems and shards run on streams that the legacy stream does not
    order: what their set-up copies and clears there has arrived when it returns, and
    before any kernel of the set-up."""
    run(fake, """
for shape in SHAPES:
    for name in OPS:
        for precision in ("fp64", "fp32"):
            for amp in (0.05, 0.0):
                op = nb.Operator(name, mesh(shape, 5, 2, amp), precision=precision)
                assert lib.fake_outstanding() == 0, (shape, name, precision, amp)
m = mesh("hex", 4, 2)
gmap, nglob, ndir = m.assembly()
ops = [nb.Operator("helmholtz", m)]
ops32 = [nb.Operator("helmholtz", m, precision="fp32")]
S = nb.GlobalLinSys(ops, gmap, nglob, ndir, sign=np.ones(len(gmap)), ops32=ops32)
assert lib.fake_outstanding() == 0
ops[0].set_wait_limit(4)
assert lib.fake_outstanding() == 0
S.set_blocks([(ndir + np.arange(3), np.eye(3))])
assert lib.fake_outstanding() == 0
S.profile(1)
assert lib.fake_outstanding() == 0
from nektar_b200.sharded import DeviceShardGroup, shard_plans
plans = shard_plans(np.asarray(gmap), ndir, 2, nc=m.nc)
nt = m.nt
halves = [nb.Operator("helmholtz", shape="hex", nm=m.nm, nq=m.nq, nelmt=4, T=m.T,
                      jac=m.jac[k:k + 4 * nt], df=np.ascontiguousarray(m.df[:, k:k + 4 * nt]),
                      deformed=True) for k in (0, 4 * nt)]
G = DeviceShardGroup(plans, [[o] for o in halves])
assert lib.fake_outstanding() == 0
assert lib.fake_early_launches() == 0
assert lib.fake_launches() > 0
""", **env)


def test_an_empty_collection_launches_nothing(fake):
    """Every operator over no elements, through every apply entry point."""
    run(fake, """
x = np.zeros(1)
for shape in SHAPES:
    m = mesh(shape, 5)
    for name in OPS:
        for precision in ("fp64", "fp32"):
            op = nb.Operator(name, shape=shape, nm=5, nq=m.nq, nelmt=0, T=m.T, jac=m.jac[:0],
                             df=np.ascontiguousarray(m.df[:, :0]), deformed=True,
                             precision=precision)
            before = lib.fake_launches()
            p = x.ctypes.data
            op.apply_device(p, p, p, p)
            if precision == "fp64":
                op(x[:0])
                if name == "iproduct_deriv":
                    op.apply3(x[:0], x[:0], x[:0])
                    op.apply3_device(p, p, p, p)
            assert lib.fake_launches() == before, (shape, name, precision)
""")


def test_an_apply_asks_the_device_nothing(fake):
    """What a launch needs to know of the device is read when the operator is created:
    two threads' first applies share nothing that either of them writes."""
    run(fake, """
x = np.zeros(1)
ops = [nb.Operator(name, mesh(shape, 4, 2)) for shape in SHAPES for name in OPS]
before = lib.fake_attribute_queries()
for op in ops:
    op.apply_device(*4 * [x.ctypes.data])
assert lib.fake_attribute_queries() == before
""")


def test_straight_sided_operators_keep_no_values_per_point(fake):
    """FP64 straight-sided operators hold 16 values per element; only LinearADR, whose
    velocities vary, packs values per point."""
    run(fake, """
for shape in SHAPES:
    for name in OPS:
        sizes = []
        for n in (2, 3):
            m, before = mesh(shape, 8, n, amp=0.0), lib.fake_allocated()
            op = nb.Operator(name, m)
            sizes.append((lib.fake_allocated() - before, m.nelmt))
        per_element = (sizes[1][0] - sizes[0][0]) / (sizes[1][1] - sizes[0][1]) / 8
        # the caller's Jacobian and nine derivative factors, and the operator's values
        assert per_element <= 10 + 16 + (10 * m.nt + 3 if name == "linear_adr" else 0), name
""")


def test_operators_name_the_kernel_that_they_run(fake):
    run(fake, """
for shape in SHAPES:
    for name in OPS:
        for nm in (4, 12):  # 13 points: beyond the line kernels
            kernel = nb.Operator(name, mesh(shape, nm)).kernel()
            assert kernel.startswith("k_line" if nm == 4 else "k_generic"), (shape, name, kernel)
""")


def test_shared_memory_is_allowed_on_every_device(fake):
    """The generic kernels' limit is raised on each device that they run on, and a small
    operator's launches and diagonal leave it for a large one's."""
    run(fake, """
x = np.zeros(1)
for shape in SHAPES:
    for device in (0, 1):
        ops = [nb.Operator("helmholtz", mesh(shape, nm), device=device) for nm in (14, 12)]
        for op in ops + ops[:1]:
            op.apply_device(x.ctypes.data, x.ctypes.data)
            op.helmholtz_diag()
            op.apply_device(x.ctypes.data, x.ctypes.data)
""", NKB_GENERIC_TUNE="0")
