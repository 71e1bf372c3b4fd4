"""Derivatives through the C ABI: Wilson action backward, the force VJP and the adjoint of
the Wilson flow, against central finite differences (FP64) and the reference's analytic
gauge force; and gradcheck through the torch.autograd binding.

Tolerances: analytic force vs action backward 1e-12; finite differences (h = 1e-5 on the
global objective, O(h^2) truncation) within 1e-6 relative to the gradient's scale; FP32 flow
gradient within 1e-3 of the FP64 one.
"""
import numpy as np
import pytest

from helpers import fail_allocations, rel

pytestmark = pytest.mark.gpu


def su2_exp_left(U, link, k, h):
    """exp(h e_k) applied from the left to one link (reference layout)."""
    from su2_b200.autograd import _exp_links
    om = np.zeros((U.size // 4, 3))
    om[link, k] = h
    return _exp_links(U, om)


def test_action_backward_is_the_reference_force(gpu, orc):
    dims, nd = (6, 4, 4, 6), 4
    U = orc.hotstart(0, dims, nd, 7, 1.0, 654321)
    with gpu.gaugeconfig(*dims, nd, 2.4) as c:
        c.upload(U)
        S, dS = c.action_backward(1.0)
    assert S == pytest.approx(orc.S_G_hmc(0, dims, nd, 2.4, U), rel=1e-12)
    assert rel(dS, orc.gauge_derivative(0, dims, nd, 2.4, U)) < 1e-12


def test_action_backward_finite_differences(gpu, orc):
    dims, nd = (4, 4, 4, 4), 4
    U = orc.hotstart(0, dims, nd, 8, 1.0, 654321)
    with gpu.gaugeconfig(*dims, nd, 2.4) as c:
        c.upload(U)
        _, dS = c.action_backward(1.0)
    rng = np.random.default_rng(1)
    for link in rng.choice(U.size // 4, 12, replace=False):
        for k in range(3):
            h = 1e-6
            fd = (orc.S_G_hmc(0, dims, nd, 2.4, su2_exp_left(U, link, k, h)) -
                  orc.S_G_hmc(0, dims, nd, 2.4, su2_exp_left(U, link, k, -h))) / (2 * h)
            assert fd == pytest.approx(dS[3 * link + k], abs=1e-6)


def test_force_vjp_finite_differences(gpu, orc):
    dims, nd = (4, 4, 4, 4), 4
    U = orc.hotstart(0, dims, nd, 9, 1.0, 654321)
    rng = np.random.default_rng(2)
    mu = rng.normal(size=U.size // 4 * 3)
    with gpu.gaugeconfig(*dims, nd, 2.0) as c:
        c.upload(U)
        vjp = c.force_vjp(mu)

    def phi(V):  # mu . g(V), g = get_deriv(U K) = derivative at beta/Nc = 1
        return float(mu @ orc.gauge_derivative(0, dims, nd, 2.0, V, 1.0, 1.0))

    for link in rng.choice(U.size // 4, 10, replace=False):
        for k in range(3):
            h = 1e-5
            fd = (phi(su2_exp_left(U, link, k, h)) - phi(su2_exp_left(U, link, k, -h))) / (2 * h)
            assert fd == pytest.approx(vjp[3 * link + k], abs=2e-6 * max(1, abs(fd)))


@pytest.mark.parametrize("dims,nd", [((6, 1, 1, 4), 2), ((2, 1, 1, 2), 2), ((4, 6, 1, 10), 3),
                                     ((6, 6, 6, 6), 4), ((2, 4, 6, 2), 4)],
                         ids=["6x4-d2", "2x2-d2", "4x6x10-d3", "6^4", "2x4x6x2"])
def test_force_vjp_geometries(gpu, orc, dims, nd):
    """The two-pass VJP in every dimension, at half volumes that are and are not whole blocks:
    central finite differences along seeded directions (FP64; O(h^2) truncation), FP32 within
    1e-5 (sums of about a hundred FP32 terms), and the buffers it borrows: the field stays, and
    the next trajectory is that of a context that took no VJP."""
    U = orc.hotstart(0, dims, nd, 9, 1.0, 654321)
    n = U.size // 4
    rng = np.random.default_rng(n)
    mu = rng.normal(size=3 * n)
    v = {}
    for prec in ("fp64", "mixed"):
        with gpu.gaugeconfig(*dims, nd, 2.0, precision=prec) as c, \
                gpu.gaugeconfig(*dims, nd, 2.0, precision=prec) as d:
            c.upload(U)
            d.upload(U)
            v[prec] = c.force_vjp(mu)
            assert np.array_equal(c.download(), d.download())
            a = c.md_update("omf2", 2, 0.5, seed=3, accept_reject=False)
            b = d.md_update("omf2", 2, 0.5, seed=3, accept_reject=False)
            assert a == b and np.array_equal(c.download(), d.download())
    assert rel(v["mixed"], v["fp64"]) < 1e-5

    from su2_b200.autograd import _exp_links

    def phi(w):
        g = orc.gauge_derivative(0, dims, nd, 2.0, _exp_links(U, w), 1.0, 1.0)
        return float(mu @ g)

    for _ in range(6):
        w = rng.normal(size=(n, 3))
        h = 1e-5
        fd = (phi(h * w) - phi(-h * w)) / (2 * h)
        scale = np.linalg.norm(v["fp64"]) * np.sqrt(3)
        assert fd == pytest.approx(float(v["fp64"] @ w.ravel()), abs=1e-6 * scale)


@pytest.mark.parametrize("dims,nd", [((6, 1, 1, 4), 2), ((4, 6, 1, 4), 3), ((4, 2, 4, 6), 4)])
def test_force_vjp_of_links_off_the_unit_sphere(gpu, orc, dims, nd):
    """An upload neither normalises nor checks: links of norm 0.7 to 1.3, some within 1e-3 and
    1e-6 of one, and a zero link.  Central differences along seeded directions as for unit links
    (their terms grow by 1.3^4 at most), FP32 within 1e-5 of FP64."""
    U = orc.hotstart(0, dims, nd, 10, 1.0, 654321)
    n = U.size // 4
    rng = np.random.default_rng(n)
    r = rng.uniform(0.7, 1.3, n)
    r[::5] = 1 + 1e-3 * rng.normal(size=r[::5].size)
    r[1::5] = 1 + 1e-6 * rng.normal(size=r[1::5].size)
    r[n // 2] = 0.0
    U = (U.reshape(n, 4) * r[:, None]).ravel()
    mu = rng.normal(size=3 * n)
    v = {}
    for prec in ("fp64", "mixed"):
        with gpu.gaugeconfig(*dims, nd, 2.0, precision=prec) as c:
            c.upload(U)
            v[prec] = c.force_vjp(mu)
    assert np.isfinite(v["mixed"]).all()
    assert rel(v["mixed"], v["fp64"]) < 1e-5
    # a global factor of the field is a factor s^4 of a force whose terms are plaquettes
    with gpu.gaugeconfig(*dims, nd, 2.0) as c:
        c.upload(1.25 * U)
        assert rel(c.force_vjp(mu), 1.25 ** 4 * v["fp64"]) < 1e-13

    from su2_b200.autograd import _exp_links

    def phi(w):
        return float(mu @ orc.gauge_derivative(0, dims, nd, 2.0, _exp_links(U, w), 1.0, 1.0))

    scale = np.linalg.norm(v["fp64"]) * np.sqrt(3)
    for _ in range(6):
        w = rng.normal(size=(n, 3))
        h = 1e-5
        fd = (phi(h * w) - phi(-h * w)) / (2 * h)
        assert fd == pytest.approx(float(v["fp64"] @ w.ravel()), abs=1e-6 * scale)


@pytest.mark.parametrize("every", [0, 1, 3])
def test_flow_adjoint_finite_differences(gpu, orc, every):
    dims, nd = (4, 4, 4, 4), 4
    U = orc.hotstart(0, dims, nd, 10, 1.0, 654321)
    eps, n = 0.02, 5
    with gpu.gaugeconfig(*dims, nd, 2.4) as c:
        c.upload(U)
        O, g = c.flow_objective(eps, n, grad=True, checkpoint_every=every)
        assert np.array_equal(c.download(), U)
        rng = np.random.default_rng(3)
        for link in rng.choice(U.size // 4, 8, replace=False):
            for k in range(3):
                h = 1e-5
                c.upload(su2_exp_left(U, link, k, h))
                Op = c.flow_objective(eps, n, grad=False)
                c.upload(su2_exp_left(U, link, k, -h))
                Om = c.flow_objective(eps, n, grad=False)
                fd = (Op - Om) / (2 * h)
                assert fd == pytest.approx(g[3 * link + k], abs=1e-7 + 1e-6 * np.abs(g).max())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,nd,n", [((4, 1, 1, 6), 2, 1), ((6, 4, 1, 4), 3, 2), ((4, 6, 4, 8), 4, 5),
                                       ((4, 4, 4, 4), 4, 30)])
def test_flow_adjoint_tape(gpu, orc, dims, nd, n, precision):
    """Every stage kept against checkpoints and recomputed stages: the same objective and
    gradient to the rounding of the stages' sums (one product and one addition, fused in one
    and not in the other), grown over 3 n stages; and the same bits from a second call."""
    U = orc.hotstart(0, dims, nd, 12, 1.0, 4321)
    tol = 3 * n * (1e-14 if precision == "fp64" else 1e-6)
    with gpu.gaugeconfig(*dims, nd, 2.4, precision=precision) as c:
        c.upload(U)
        O, g = c.flow_objective(0.02, n)
        O2, g2 = c.flow_objective(0.02, n)
        assert O == O2 and np.array_equal(g, g2)
        for every in (1, 3):
            Oc, gc = c.flow_objective(0.02, n, checkpoint_every=every)
            assert O == pytest.approx(Oc, rel=tol)
            assert np.linalg.norm(g - gc) <= tol * np.linalg.norm(gc)
        assert c.flow_objective(0.02, n, grad=False) == pytest.approx(O, rel=tol)


def test_flow_adjoint_tape_limit(gpu, orc):
    """More steps than the tape may hold (8 GB: about 3,100 steps of an 8^4 FP64 lattice) take
    the checkpoints that they took without it: the bits of the explicit choice."""
    dims, n = (8, 8, 8, 8), 3200
    U = orc.hotstart(0, dims, 4, 13, 1.0, 4321)
    with gpu.gaugeconfig(*dims, 4, 2.4) as c:
        c.upload(U)
        O, g = c.flow_objective(1e-4, n)
        Oc, gc = c.flow_objective(1e-4, n, checkpoint_every=round(n ** 0.5))
        assert O == Oc and np.array_equal(g, gc)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_flow_adjoint_without_memory_for_the_tape(gpu, orc, precision):
    """A tape whose allocation is refused: the gradient of the checkpoints, bit for bit, in the
    same call.  Refused both: an error, and the next call is none the worse."""
    dims, n = (4, 6, 4, 8), 9
    U = orc.hotstart(0, dims, 4, 14, 1.0, 4321)
    with gpu.gaugeconfig(*dims, 4, 2.4, precision=precision) as c:
        c.upload(U)
        fail_allocations(c, 1)
        O, g = c.flow_objective(0.02, n)
        Oc, gc = c.flow_objective(0.02, n, checkpoint_every=3)
        assert O == Oc and np.array_equal(g, gc)
    with gpu.gaugeconfig(*dims, 4, 2.4, precision=precision) as c:
        c.upload(U)
        fail_allocations(c, 2)
        with pytest.raises(gpu.Su2bError, match="scratch"):
            c.flow_objective(0.02, n)
        assert np.isfinite(c.gauge_energy())
        assert c.flow_objective(0.02, n)[0] == pytest.approx(Oc, rel=1e-5)


def free_bytes():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def test_tape_memory_is_given_back(gpu, orc):
    """The stages of 20 steps at 16^4 FP64 are 0.88 GB: they stay for the next gradient, and go
    when a call asks for checkpoints, when another context finds no memory and when the context
    ends; the gradients after that are those before.  The device allocates in pieces of 2 MB."""
    dims, n, piece = (16, 16, 16, 16), 20, 4 << 20
    tape = 3 * n * 4 * 16 ** 4 * (32 + 24)
    U = orc.hotstart(0, dims, 4, 15, 1.0, 4321)
    with gpu.gaugeconfig(*dims, 4, 2.4) as c, gpu.gaugeconfig(4, 1, 1, 4, 2, 2.4) as other:
        c.upload(U)
        c.flow_objective(0.01, n, checkpoint_every=5)
        before = free_bytes()
        want = c.flow_objective(0.01, n)
        assert before - free_bytes() > tape // 2
        held = free_bytes()
        for k in range(2):
            got = c.flow_objective(0.01, n)
            assert got[0] == want[0] and np.array_equal(got[1], want[1])
        assert free_bytes() == held
        c.flow_objective(0.01, n, checkpoint_every=5)
        assert abs(free_bytes() - before) <= piece
        got = c.flow_objective(0.01, n)
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
        fail_allocations(other, 1)
        with pytest.raises(gpu.Su2bError):
            other.flow_objective(0.01, 2, checkpoint_every=1)
        assert free_bytes() >= before - piece
        got = c.flow_objective(0.01, n)
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
        assert before - free_bytes() > tape // 2
        c.close()
        assert free_bytes() > before


def test_tapes_of_all_contexts_share_one_limit(gpu, orc):
    """Two contexts whose stages take 5 GB each: the second one's gradient is the checkpoints',
    bit for bit, until the first context ends."""
    dims, n = (16, 16, 16, 16), 114
    U = orc.hotstart(0, dims, 4, 16, 1.0, 4321)
    with gpu.gaugeconfig(*dims, 4, 2.4) as b:
        b.upload(U)
        with gpu.gaugeconfig(*dims, 4, 2.4) as a:
            a.upload(U)
            a.flow_objective(1e-3, n)
            before = free_bytes()
            O, g = b.flow_objective(1e-3, n)
            assert before - free_bytes() < 1 << 30
            Oc, gc = b.flow_objective(1e-3, n, checkpoint_every=round(n ** 0.5))
            assert O == Oc and np.array_equal(g, gc)
        before = free_bytes()
        O, g = b.flow_objective(1e-3, n)
        assert before - free_bytes() > 4 << 30
        assert O == pytest.approx(Oc, rel=1e-11)


def test_flow_objective_matches_flow_records(gpu, orc):
    dims, nd = (4, 4, 4, 4), 4
    U = orc.hotstart(0, dims, nd, 11, 1.0, 654321)
    Vt = U.copy()
    for _ in range(4):
        Vt = orc.runge_kutta(0, dims, nd, 2.4, 0.02, Vt)
    P = orc.gauge_energy(0, dims, nd, Vt) / (256 * 2)
    want = (4 * 0.02) ** 2 * (6 - P)
    with gpu.gaugeconfig(*dims, nd, 2.4) as c:
        c.upload(U)
        assert c.flow_objective(0.02, 4, grad=False) == pytest.approx(want, rel=1e-12)


def test_flow_adjoint_fp32_against_fp64(gpu, orc):
    dims, nd = (8, 8, 8, 8), 4
    U = orc.hotstart(0, dims, nd, 12, 1.0, 654321)
    res = {}
    for prec in ("fp64", "mixed"):
        with gpu.gaugeconfig(*dims, nd, 2.4, precision=prec) as c:
            c.upload(U)
            res[prec] = c.flow_objective(0.01, 20, grad=True)
    assert res["mixed"][0] == pytest.approx(res["fp64"][0], rel=1e-5)
    assert rel(res["mixed"][1], res["fp64"][1]) < 1e-3


def test_autograd_binding_gradcheck(gpu, orc):
    import torch

    from su2_b200.autograd import FlowEnergy, WilsonAction
    dims, nd = (2, 2, 2, 4), 4
    U = orc.hotstart(0, dims, nd, 13, 1.0, 654321)
    n = U.size // 4
    with gpu.gaugeconfig(*dims, nd, 2.3) as c:
        om = (0.05 * torch.randn(n, 3, dtype=torch.float64)).requires_grad_()
        assert torch.autograd.gradcheck(lambda w: WilsonAction.apply(w, c, U), (om,), eps=1e-6,
                                        atol=1e-6, rtol=1e-5)
        assert torch.autograd.gradcheck(lambda w: FlowEnergy.apply(w, c, U, 0.05, 3, 2), (om,),
                                        eps=1e-6, atol=1e-7, rtol=1e-5)
