"""The one-launch stage of the linear Ch operator (SBP 4-2) against the CPU FP64 oracle.

Every tile computes the neighbour panels' boundary values it needs itself, so the cube
sizes put the panel's far edge at every position within a vector of points (four FP32, two
FP64), with one, two and several tiles per direction.  Random states: the duplicated edge
vertices and both winds disagree across the panels.  Tolerances as for the other stage
kernels: FP64 within 1e-12 relative (max-norm) of the oracle, FP32 within 1e-5.
"""
import functools

import numpy as np
import pytest

from ch_swe_b200._lib import SweError
from tests.conftest import gpu_available

pytestmark = pytest.mark.gpu

LIN = {"swm_operator_type": "linear_swm_operator", "h_mean": 1000.0}
CFGS = [("fp64", c) for c in ((17, 1, 3), (25, 1, 3), (33, 1, 3))] + [("fp32", c) for c in ((17, 2, 3), (25, 2, 3), (33, 2, 3))]
RTOL = {"fp64": 1e-12, "fp32": 1e-5}


@pytest.fixture(scope="module", autouse=True)
def _need_gpu(lib_built, oracle_built):
    if not gpu_available():
        pytest.fail("no CUDA device: the -m gpu tests need a B200")


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def random_state(N, seed):
    from ch_swe_b200 import state_shapes
    rng = np.random.default_rng(seed)
    return tuple(rng.standard_normal(s) for s in state_shapes(N))


AXIS = (0.3, -0.5, 0.8)


@functools.lru_cache(maxsize=None)
def linear_reference(N):
    """A random state and the oracle's tendency, shared by the configurations."""
    from oracle.oracle import Oracle
    state = random_state(N, 900 + N)
    return state, Oracle(N, h_mean=1000.0, axis=AXIS).apply(*state)


@pytest.mark.parametrize("precision,cfg", CFGS)
@pytest.mark.parametrize("N", [8, 9, 10, 11, 16, 21, 23, 24, 31, 32, 33, 34, 46, 48, 65, 79, 150])
def test_apply_matches_oracle(precision, cfg, N):
    """Up to more blocks than the device takes at once (C150).  FP64 configurations whose
    blocks touch too many sides for the register file are refused: all of them where one tile
    spans the panel both ways, the largest also where one spans it in one direction."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator
    (h, u, v), ref = linear_reference(N)
    dom = create_domain(N, precision=precision, h_mean=1000.0, rotation_axis=AXIS)
    if precision == "fp64" and (N <= 11 or (cfg == (33, 1, 3) and N <= 24)):
        with pytest.raises(SweError):
            dom.kernel_config = cfg
        dom.destroy()
        return
    dom.kernel_config = cfg
    assert dom.kernel_config == cfg
    op = create_swm_operator(dom.grav, LIN, dom)
    x, y = create_stvec_swm(dom).upload(h, u, v), create_stvec_swm(dom)
    op.apply(y, x, dom)
    dom.synchronize()
    for g, r, name in zip(y.download(), ref, "huv"):
        assert rel(g, r) < RTOL[precision], (name, rel(g, r))
    dom.destroy()


@pytest.mark.parametrize("precision,cfg", CFGS)
def test_rk4_members_match_the_split_stage(precision, cfg):
    """Steps with a time step per member (one frozen) and a mean depth per member agree with
    the split kernels to rounding; the zero margins and the frozen member stay as they were."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    N, M = 37, 3
    states = [random_state(N, 40 + k) for k in range(M)]
    stack = [np.stack([s[f] for s in states]) for f in range(3)]
    dts = np.array([300.0, 0.0, 150.0])
    out = []
    for c in (cfg, (25, 2, 0)):
        dom = create_domain(N, precision=precision, n_members=M, h_mean=1000.0)
        dom.kernel_config = c
        op = create_swm_operator(dom.grav, LIN, dom)
        op.set_member_h_mean(2, 700.0)
        st = create_stvec_swm(dom).upload(*stack, member=None)
        create_timescheme(st, "rk4").steps_members(st, op, dts, 11)
        dom.synchronize()
        out.append(st.download(member=None))
        dom.destroy()
    for f in range(3):
        assert rel(out[0][f], out[1][f]) < RTOL[precision]
        assert np.array_equal(out[0][f][1], stack[f][1].astype(np.float32 if precision == "fp32" else np.float64))


def test_default_stage_matches_oracle_and_joins_a_group():
    """A linear context that sets no configuration runs the one-launch stage; a group takes it
    with its split configuration."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    from ch_swe_b200.swm import create_group
    from oracle.oracle import Oracle
    N, dt = 100, 200.0
    o = Oracle(N, h_mean=1000.0)
    ic = o.gaussian(lam0=0.7, phi0=0.2, d0=0.2)
    ref = o.rk4(*ic, dt, 3)
    dom = create_domain(N, h_mean=1000.0)
    assert dom.kernel_config[2] == 3 and dom.tile == 33
    op = create_swm_operator(dom.grav, LIN, dom)
    st = create_stvec_swm(dom).upload(*ic)
    create_timescheme(st, "rk4").steps(st, op, dom, dt, 3)
    for g, r in zip(st.download(), ref):
        assert rel(g, r) < 1e-12
    st.upload(*ic)
    g = create_group([dom])
    g.steps_members([st], [np.array([dt])], 3)
    g.synchronize()
    for a, r in zip(st.download(), ref):
        assert rel(a, r) < 1e-12
    g.destroy()
    dom.destroy()


ADV_CFGS = [("fp64", c) for c in ((17, 2, 3), (25, 2, 3), (33, 1, 3))] + [("fp32", c) for c in ((25, 2, 3), (33, 2, 3))]


@pytest.mark.parametrize("orography", [False, True])
@pytest.mark.parametrize("precision,cfg", ADV_CFGS)
@pytest.mark.parametrize("N", [16, 23, 24, 31, 33, 34, 46, 65, 79])
def test_advective_apply_matches_oracle(precision, cfg, N, orography):
    """The advective operator's vector kernels: random winds and disagreeing edge copies on a
    full depth, with and without orography."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator
    from oracle.oracle import Oracle
    rng = np.random.default_rng(70 + N)
    h, u, v = random_state(N, 300 + N)
    h = 1000.0 + 50.0 * h
    hs = 100.0 * rng.standard_normal(h.shape) if orography else None
    axis = (0.3, -0.5, 0.8)
    o = Oracle(N, axis=axis, operator="advective")
    if orography:
        o.set_orography(hs)
    ref = o.apply(h, u, v)
    dom = create_domain(N, precision=precision, rotation_axis=axis, operator="advective")
    dom.kernel_config = cfg
    assert dom.kernel_config == cfg
    op = create_swm_operator(dom.grav, {"swm_operator_type": "advective_swm_operator"}, dom)
    if orography:
        op.set_orography(hs)
    x, y = create_stvec_swm(dom).upload(h, u, v), create_stvec_swm(dom)
    op.apply(y, x, dom)
    dom.synchronize()
    for g, r, name in zip(y.download(), ref, "huv"):
        assert rel(g, r) < RTOL[precision], (name, rel(g, r))
    dom.destroy()


@pytest.mark.parametrize("cfg", [(25, 2, 0), (25, 2, 3)])
@pytest.mark.parametrize("N", [22, 23])
def test_advective_members_share_the_halo_launch(N, cfg):
    """Edge averages and virtual winds of all members in one launch: 252 edge vertices fit one
    block of a member, 264 need two; member 1 is frozen."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    from oracle.oracle import Oracle
    M = 3
    states = [random_state(N, 600 + 10 * N + k) for k in range(M)]
    stack = [np.stack([s[f] + (0.0 if f else 1000.0) for s in states]) for f in range(3)]
    dts = np.array([60.0, 0.0, 30.0])
    dom = create_domain(N, n_members=M, operator="advective")
    dom.kernel_config = cfg
    op = create_swm_operator(dom.grav, {"swm_operator_type": "advective_swm_operator"}, dom)
    st = create_stvec_swm(dom).upload(*stack, member=None)
    create_timescheme(st, "rk4").steps_members(st, op, dts, 2)
    dom.synchronize()
    out = st.download(member=None)
    o = Oracle(N, operator="advective")
    for m in (0, 2):
        ref = o.rk4(*(f[m] for f in stack), dts[m], 2)
        for g, r, name in zip(out, ref, "huv"):
            assert rel(g[m], r) < 1e-12, (m, name, rel(g[m], r))
    for f in range(3):
        assert np.array_equal(out[f][1], stack[f][1])
    dom.destroy()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("operator", ["linear", "advective"])
@pytest.mark.parametrize("N", [8, 9, 10, 11, 12, 13, 14, 15])
def test_default_stage_of_the_smallest_cubes(N, operator, precision):
    """Below 16 cells too a context starts on the vector stage where a configuration's blocks fit
    (linear FP64: from 13 cells on); members with their own time steps against the oracle."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    from oracle.oracle import Oracle
    M = 2
    states = [random_state(N, 10 * N + k) for k in range(M)]
    stack = [np.stack([s[f] + (1000.0 if operator == "advective" and f == 0 else 0.0) for s in states]) for f in range(3)]
    dts = np.array([60.0, 30.0])
    dom = create_domain(N, precision=precision, n_members=M, operator=operator, h_mean=1000.0)
    assert (dom.kernel_config[2] == 3) == (operator == "advective" or precision == "fp32" or N >= 13)
    op = create_swm_operator(dom.grav, {"swm_operator_type": operator + "_swm_operator", "h_mean": 1000.0}, dom)
    st = create_stvec_swm(dom).upload(*stack, member=None)
    create_timescheme(st, "rk4").steps_members(st, op, dts, 3)
    dom.synchronize()
    out = st.download(member=None)
    o = Oracle(N, h_mean=1000.0, operator=operator)
    for m in range(M):
        ref = o.rk4(*(f[m] for f in stack), dts[m], 3)
        for g, r, name in zip(out, ref, "huv"):
            assert rel(g[m], r) < RTOL[precision], (m, name, rel(g[m], r))
    dom.destroy()


@pytest.mark.parametrize("operator,precision,N,members,cfg", [
    ("linear", "fp64", 18, 16, (25, 1, 3)), ("linear", "fp64", 22, 16, (17, 1, 3)), ("linear", "fp64", 22, 24, (25, 1, 3)), ("linear", "fp64", 18, 64, (25, 1, 3)), ("linear", "fp64", 12, 64, (25, 2, 0)), ("linear", "fp64", 24, 64, (25, 1, 3)),
    ("linear", "fp64", 26, 64, (17, 1, 3)), ("linear", "fp64", 96, 1, (25, 1, 3)), ("linear", "fp64", 192, 1, (33, 1, 3)),
    ("linear", "fp32", 192, 1, (33, 2, 3)), ("advective", "fp64", 108, 1, (33, 1, 3)), ("advective", "fp64", 128, 1, (17, 2, 3)),
    ("advective", "fp64", 64, 4, (25, 2, 3)), ("advective", "fp64", 80, 16, (17, 2, 3)), ("advective", "fp32", 52, 1, (33, 2, 3)), ("advective", "fp32", 80, 1, (25, 2, 3)),
    ("advective", "fp32", 80, 4, (33, 2, 3)), ("advective", "fp32", 128, 1, (33, 2, 3))])
def test_default_configuration(operator, precision, N, members, cfg):
    """The configuration a context starts with, on both sides of each line of the rule: the
    sizes at which another one was measured slower are among them."""
    from ch_swe_b200 import create_domain
    dom = create_domain(N, precision=precision, n_members=members, operator=operator)
    assert dom.kernel_config == cfg
    dom.destroy()


@pytest.mark.parametrize("orography", [False, True])
@pytest.mark.parametrize("precision,cfg", ADV_CFGS)
def test_advective_members_of_every_configuration(precision, cfg, orography):
    """RK4 steps of three members (own time steps, one frozen) with several tiles per direction,
    against the oracle: the RK modes, the FP32 update's compensation and the FP32 tendencies."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    from oracle.oracle import Oracle
    N, M = 66, 3
    states = [random_state(N, 800 + k) for k in range(M)]
    stack = [np.stack([s[f] + (0.0 if f else 1000.0) for s in states]) for f in range(3)]
    dts = np.array([30.0, 0.0, 15.0])
    hs = 100.0 * np.random.default_rng(9).standard_normal(stack[0][0].shape) if orography else None
    dom = create_domain(N, precision=precision, n_members=M, operator="advective")
    dom.kernel_config = cfg
    op = create_swm_operator(dom.grav, {"swm_operator_type": "advective_swm_operator"}, dom)
    o = Oracle(N, operator="advective")
    if orography:
        op.set_orography(hs)
        o.set_orography(hs)
    st = create_stvec_swm(dom).upload(*stack, member=None)
    create_timescheme(st, "rk4").steps_members(st, op, dts, 3)
    dom.synchronize()
    out = st.download(member=None)
    for m in (0, 2):
        for g, r, name in zip(out, o.rk4(*(f[m] for f in stack), dts[m], 3), "huv"):
            assert rel(g[m], r) < RTOL[precision], (m, name, rel(g[m], r))
    for f in range(3):
        assert np.array_equal(out[f][1], stack[f][1].astype(np.float32 if precision == "fp32" else np.float64))
    dom.destroy()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("N,members", [(12, 16), (13, 16), (14, 64), (16, 16), (16, 64), (18, 128), (24, 64), (30, 48)])
def test_members_have_the_bits_of_single_contexts(N, members, precision):
    """Whether a cube starts on the vector stage does not depend on its number of members, and
    every tile shape gives the same bits: a member's are those of a context of its own."""
    from ch_swe_b200 import create_domain, create_stvec_swm, create_swm_operator, create_timescheme
    states = [random_state(N, 20 + k) for k in range(3)]
    picked = {0: 0, members // 2: 1, members - 1: 2}
    out = []
    for M in (members, 1, 1, 1):
        dom = create_domain(N, precision=precision, n_members=M, h_mean=1000.0)
        op = create_swm_operator(dom.grav, LIN, dom)
        st = create_stvec_swm(dom)
        for m, k in picked.items() if M > 1 else ((0, len(out) - 1),):
            st.upload(*states[k], member=m)
        create_timescheme(st, "rk4").steps(st, op, dom, 100.0, 3)
        out.append([st.download(member=m) for m in (picked if M > 1 else (0,))])
        dom.destroy()
    for k in range(3):
        for a, b in zip(out[0][k], out[1 + k][0]):
            assert np.array_equal(a, b)
