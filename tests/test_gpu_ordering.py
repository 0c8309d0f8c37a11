"""Work of a context against work of others on the default stream.

A context's stream does not wait for the default stream, where a host program may have
kernels of its own queued (torch's current stream is that one).  Buffers cleared or tables
copied there are late whenever it is busy: here it is kept busy while a context is created,
its state uploaded and advanced, and while the diagnostics build their tables on first use.
Every result has the bits that it has on an idle device.
"""
import numpy as np
import pytest

from tests.conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(lib_built, oracle_built):
    if not gpu_available():
        pytest.fail("no CUDA device: the -m gpu tests need a B200")


def busy():
    """About 20 ms of work queued on the default stream."""
    import torch
    torch.cuda._sleep(40_000_000)


def idle():
    import torch
    torch.cuda.synchronize()


def make(N, wait, **kw):
    """A context, its operator and a state that holds a random upload, `wait` before every step."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator
    from ch_swe_b200.swm import state_shapes
    rng = np.random.default_rng(N)
    ic = [rng.standard_normal(s) for s in state_shapes(N, None, kw.get("horizontal_staggering", "Ch"))]
    if kw.get("operator") == "advective":
        ic[0] += 1000.0
    wait()
    dom = create_domain(N, h_mean=1000.0, **kw)
    op = create_swm_operator(dom.grav, {"swm_operator_type": "advective_swm_operator"} if kw.get("operator") == "advective"
                             else {"swm_operator_type": "linear_swm_operator", "h_mean": 1000.0}, dom)
    wait()
    return ic, dom, op, create_stvec_swm(dom).upload(*ic)


CONTEXTS = [dict(), dict(precision="fp32"), dict(operator="advective"), dict(operator="advective", precision="fp32"),
            dict(sbp_order=21), dict(horizontal_staggering="Ah"), dict(horizontal_staggering="Ah", diffusion=42)]


@pytest.mark.parametrize("kw", CONTEXTS, ids=lambda k: "-".join(str(v) for v in k.values()) or "linear")
@pytest.mark.parametrize("N", [24, 89])
def test_first_pass_of_a_fresh_context(N, kw):
    from ch_swe_b200 import create_timescheme
    from ch_swe_b200.swm import create_swm_diff_operator
    from oracle.oracle import Oracle
    kw = dict(kw)
    order = kw.pop("diffusion", 0)
    out = []
    for wait in (idle, busy, busy):
        ic, dom, op, st = make(N, wait, **kw)
        mass = op.integrals(st)
        if order:
            wait()
            dom.set_diffusion(create_swm_diff_operator(
                {"hordiff_uv_name": f"hordiff_vec_xyz_Ah_sbp_{order}_narrow", "uv_diff_coeff": 0.03,
                 "hordiff_h_name": f"hordiff_scalar_Ah_sbp_{order}_narrow", "h_diff_coeff": 0.01}, dom))
        create_timescheme(st, "rk4").steps(st, op, dom, 10.0, 3)
        out.append([np.array(mass), *st.download()])
        idle()
        dom.destroy()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
    if not kw:
        for g, r in zip(out[1][1:], Oracle(N, h_mean=1000.0).rk4(*ic, 10.0, 3)):
            assert np.abs(g - r).max() < 1e-12 * np.abs(r).max()


@pytest.mark.parametrize("what", ["curl", "energies", "h", "div", "regrid_curl", "wind"])
@pytest.mark.parametrize("N", [8, 24])
def test_tables_of_the_diagnostics_on_first_use(N, what):
    from ch_swe_b200.diag import LatlonOutputer, LatlonVecOutputer, SwmOutputDiag
    out = []
    for wait in (idle, busy):
        _, dom, _, st = make(N, wait)
        idle()
        wait()
        if what == "curl":
            r = [SwmOutputDiag(dom).curl(st)]
        elif what == "energies":
            r = [np.array(list(SwmOutputDiag(dom).calc_energies(st).values()))]
        elif what == "wind":
            r = list(LatlonVecOutputer(dom, 8, 16).regrid(st))
        else:
            r = [getattr(LatlonOutputer(dom, 8, 16), {"h": "regrid"}.get(what, what if what.startswith("regrid") else "regrid_" + what))(st)]
        out.append([np.array(a) for a in r])
        idle()
        dom.destroy()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_synchronize_waits_for_the_default_stream():
    """A state written through its device view by work on the default stream is in place after
    swe_synchronize, for the context's stream."""
    import math
    import torch
    ic, dom, _, st = make(16, idle)
    ptr, nbytes, _, _ = st.device_view()

    class View:
        __cuda_array_interface__ = {"data": (ptr, False), "shape": (nbytes // 8,), "typestr": "<f8", "version": 3}

    box = torch.as_tensor(View(), device="cuda")
    assert math.prod(box.shape) * 8 == nbytes
    box.mul_(1.0)   # the kernel is loaded
    idle()
    busy()
    box.mul_(2.0)
    dom.synchronize()
    for a, b in zip(ic, st.download()):
        assert np.array_equal(2.0 * a, b)
    idle()
    del box, st
    dom.destroy()
