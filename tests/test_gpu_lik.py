"""GPU log-likelihood forward pass and adjoint against the FP64 oracle.

The GPU computes each weight in fp32 (one exp2 of an exponent carried as an fp32 pair) and every
normaliser and log-sum in FP64 or compensated fp32; the oracle is FP64 throughout.  Tolerances:
log-likelihood relative error <= 1e-7 (fp32 weights carry about 1e-7 relative error into each of
the ~1e5 terms); gradient relative error (2-norm over the four components) <= 1e-6 at the 64
points drawn from the parameter ranges.  At the generating point theta* the gradient is close to
zero -- the trace was drawn there -- so errors that do not average out over the trace are a larger
share of it: the default arithmetic (special-function-unit exp2, pairwise ball sums) is held to
1e-5 there, the exact arithmetic (pg_lik_set_exact_exp2) to 1e-6 like every other point."""
import math

import numpy as np
import pytest

import oracle as O
from paragraph_gb300 import GrowthEngine, PGError, TraceInput
from paragraph_gb300 import workloads as W

pytestmark = pytest.mark.gpu
THETA_STAR = np.array([1.0, 5.0, 1.0, 4.0])


@pytest.fixture(scope="module")
def trace_mid(gpu):
    g = W.plain_pa_seed(20_000, 10, seed=3)
    return W.grow_trace(g, W.calibration_params(), 10, seed=5)


def test_gpu_trace_equals_oracle_trace(gpu):
    """Anchors and draw-order citations recorded by the GPU growth step match the oracle's."""
    g = W.plain_pa_seed(4000, 10, seed=4)
    prm = W.calibration_params()
    tg = W.grow_trace(g, prm, 4, seed=9)
    to = O.grow_trace(g, prm, 4, seed=9)
    for f in ("epoch_nodes", "epoch_t", "anchors", "cite_off", "cites", "pub"):
        np.testing.assert_array_equal(getattr(tg, f), getattr(to, f), err_msg=f)
    np.testing.assert_array_equal(tg.fitness.view(np.uint32), to.fitness.view(np.uint32))


def test_loglik_and_gradient_match_fp64_oracle(trace_mid):
    pts = np.vstack([THETA_STAR, W.theta_batch(64, seed=1)])
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(trace_mid)
        ll = eng.loglik(pts)
        gr = eng.loglik_grad(pts)
    llo, gro = O.loglik(trace_mid, pts)
    rel_ll = np.abs(ll - llo) / np.abs(llo)
    rel_g = np.linalg.norm(gr - gro, axis=1) / np.linalg.norm(gro, axis=1)
    msg = f"loglik {rel_ll.max():.3g}, grad (64 points) {rel_g[1:].max():.3g}, grad (theta*) {rel_g[0]:.3g}"
    print(msg)
    assert rel_ll.max() <= 1e-7, msg
    assert rel_g[1:].max() <= 1e-6, msg
    assert rel_g[0] <= 1e-5, msg


def test_exact_arithmetic_meets_1e6_at_the_generating_point(trace_mid):
    """The exact arithmetic (fp32 exp2 to ~2 ulp, every ball weight and product summed on its own)
    holds the gradient within 1e-6 of the FP64 oracle at theta* as well, in batches of one point
    (the sliced ball walk) and of nine (one lane per point)."""
    pts = np.vstack([THETA_STAR, W.theta_batch(8, seed=11)])
    llo, gro = O.loglik(trace_mid, pts)
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(trace_mid)
        eng.set_lik_exact_exp2(True)
        ll = eng.loglik(pts)
        gr = eng.loglik_grad(pts)
        l1 = eng.loglik(pts[:1])
        g1 = eng.loglik_grad(pts[:1])
    rel_ll = np.abs(ll - llo) / np.abs(llo)
    rel_g = np.linalg.norm(gr - gro, axis=1) / np.linalg.norm(gro, axis=1)
    rel_1 = np.linalg.norm(g1[0] - gro[0]) / np.linalg.norm(gro[0])
    msg = f"loglik {rel_ll.max():.3g}, grad (theta*) {rel_g[0]:.3g} / alone {rel_1:.3g}, others {rel_g[1:].max():.3g}"
    assert rel_ll.max() <= 1e-7 and abs(l1[0] - llo[0]) <= 1e-7 * abs(llo[0]), msg
    assert rel_g.max() <= 1e-6 and rel_1 <= 1e-6, msg


def test_arithmetic_modes_switch_cleanly(trace_mid):
    """The feature rows follow the arithmetic of each forward pass and the adjoint keeps the
    forward's: default results after exact passes, with the mode switched again before the adjoint,
    equal a fresh context's default results bit for bit."""
    pts = W.theta_batch(3, seed=13)
    with GrowthEngine(seed=1) as a, GrowthEngine(seed=1) as b:
        a.load_trace(trace_mid)
        b.load_trace(trace_mid)
        l0 = a.loglik(pts)
        g0 = a.loglik_grad(pts)
        b.set_lik_exact_exp2(True)
        lx = b.loglik(pts)
        b.loglik_grad(pts)
        b.set_lik_exact_exp2(False)
        l1 = b.loglik(pts)
        b.set_lik_exact_exp2(True)
        g1 = b.loglik_grad(pts)
    np.testing.assert_array_equal(l0, l1)
    np.testing.assert_array_equal(g0, g1)
    assert not np.array_equal(l0, lx)


def test_batch_groups_and_single_points_agree(trace_mid):
    """70 points run as two launches of <= 64; every point alone gives the same values.  A single
    point splits the ball sums over more threads than a batch, so the compensated fp32 partial
    sums differ in order: agreement is to 1e-9 (log-likelihood) and 1e-7 (gradient), not bitwise."""
    pts = W.theta_batch(70, seed=2)
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(trace_mid)
        ll = eng.loglik(pts)
        gr = eng.loglik_grad(pts, dloglik=np.full(70, 2.0))
        for b in (0, 33, 64, 69):
            l1 = eng.loglik(pts[b:b + 1])
            g1 = eng.loglik_grad(pts[b:b + 1])
            assert abs(l1[0] - ll[b]) <= 1e-9 * abs(ll[b])
            assert np.linalg.norm(2.0 * g1[0] - gr[b]) <= 1e-7 * np.linalg.norm(gr[b])


def test_adjoint_matches_gpu_central_differences(trace_mid):
    """Central differences of the GPU's own log-likelihood (h = 1e-4).  The fp32 weights make the
    log-likelihood accurate to about 1e-8 relative, about 1e-2 absolute here, and that rounding
    changes from one point to the next, so the differences carry up to 1e-2 / 2e-4 = 50 units of
    noise on gradients of 1e4: the check is at 1e-3 relative.  The FP64 gradient of the oracle
    meets central differences at 1e-6 (tests/test_lik_oracle.py) and the GPU adjoint meets that
    FP64 gradient at 1e-6 (above)."""
    pts = W.theta_batch(4, seed=5)
    h = 1e-4
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(trace_mid)
        eng.loglik(pts)
        gr = eng.loglik_grad(pts)
        for b in range(len(pts)):
            shifted = []
            for k in range(4):
                for s in (1.0, -1.0):
                    t = pts[b].copy()
                    t[k] += s * h
                    shifted.append(t)
            l = eng.loglik(np.array(shifted))
            fd = (l[0::2] - l[1::2]) / (2 * h)
            assert np.linalg.norm(fd - gr[b]) / np.linalg.norm(gr[b]) <= 1e-3


def test_adjoint_needs_the_forward_points(trace_mid):
    pts = W.theta_batch(3, seed=8)
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(trace_mid)
        with pytest.raises(PGError):
            eng.loglik_grad(pts)
        eng.loglik(pts)
        with pytest.raises(PGError):
            eng.loglik_grad(pts[:2])
        eng.loglik_grad(pts)


def test_ball_bitmap_in_several_passes(gpu):
    """A seed of 900k nodes needs two shared-memory bitmap passes (786,432 ids each)."""
    g = W.plain_pa_seed(900_000, 10, seed=6)
    prm = W.calibration_params()
    prm.growth_rate = 0.0
    prm.fixed_new_nodes = 3000
    tr = W.grow_trace(g, prm, 1, seed=2)
    pts = np.vstack([THETA_STAR, [0.7, 3.0, 1.5, 6.0]])
    with GrowthEngine(seed=1) as eng:
        eng.load_trace(tr)
        ll = eng.loglik(pts)
        gr = eng.loglik_grad(pts)
    llo, gro = O.loglik(tr, pts)
    assert (np.abs(ll - llo) / np.abs(llo)).max() <= 1e-7
    rel = np.linalg.norm(gr - gro, axis=1) / np.linalg.norm(gro, axis=1)
    assert rel[0] <= 1e-5 and rel[1] <= 1e-6, rel


def test_ball_chunks_rebuilt_per_pass_give_identical_results(trace_mid):
    """Balls kept for all agents at once, or rebuilt chunk by chunk in every pass (what a trace too
    large for memory does): the per-agent arithmetic is the same, so the results are bitwise equal."""
    pts = W.theta_batch(5, seed=4)
    with GrowthEngine(seed=1) as a, GrowthEngine(seed=1) as b:
        a.load_trace(trace_mid)
        b.set_tuning(lik_chunk_agents=700)
        b.load_trace(trace_mid)
        la, lb = a.loglik(pts), b.loglik(pts)
        ga, gb = a.loglik_grad(pts), b.loglik_grad(pts)
    np.testing.assert_array_equal(la, lb)
    np.testing.assert_array_equal(ga, gb)


def _check_against_oracle(trace, pts, exact=False):
    """Log-likelihood to 1e-7, gradient to 1e-6: the bounds stated at the top of this file."""
    with GrowthEngine(seed=1) as eng:
        eng.set_lik_exact_exp2(exact)
        eng.load_trace(trace)
        ll, gr = eng.loglik(pts), eng.loglik_grad(pts)
        balls = eng.stats()["lik_ball_elems"]
    llo, gro = O.loglik(trace, pts)
    assert (np.abs(ll - llo) / np.abs(llo)).max() <= 1e-7
    assert (np.linalg.norm(gr - gro, axis=1) / np.linalg.norm(gro, axis=1)).max() <= 1e-6
    return balls, int(trace.epoch_nodes[:-1].sum())


@pytest.mark.parametrize("points", [1, 2, 3, 8, 9, 16, 17, 32, 33, 63, 64, 65])
def test_weight_table_at_every_row_width(gpu, points):
    """Balls summed from the weight table: every lane layout (points a power of two, one above, one
    below), balls of all remainders (a 2-hop ball's size is arbitrary), agents of several epochs."""
    g = W.plain_pa_seed(1500, 6, seed=21)
    tr = W.grow_trace(g, W.calibration_params(), 3, seed=5)
    balls, rows = _check_against_oracle(tr, W.theta_batch(points, seed=points), exact=points % 2 == 1)
    assert balls >= 4 * rows  # the table is used at every batch size


def test_weights_evaluated_in_place_for_few_balls(gpu):
    """Few ball elements for the nodes there are: no table."""
    g = W.plain_pa_seed(60_000, 3, seed=22)
    prm = W.calibration_params()
    prm.growth_rate, prm.fixed_new_nodes = 0.0, 40
    tr = W.grow_trace(g, prm, 2, seed=6)
    for points in (2, 40):
        balls, rows = _check_against_oracle(tr, W.theta_batch(points, seed=points))
        assert 8 * balls < rows


def test_weight_table_in_several_parts(gpu):
    """Four epochs of 1.1M nodes: the table holds three of them at a time (1 GiB at 64 points)."""
    g = W.plain_pa_seed(1_100_000, 10, seed=23)
    prm = W.calibration_params()
    prm.growth_rate, prm.fixed_new_nodes = 0.0, 2500
    tr = W.grow_trace(g, prm, 4, seed=7)
    balls, rows = _check_against_oracle(tr, W.theta_batch(3, seed=9))
    assert 8 * balls >= rows


def _unit_weight_trace(nodes, cites):
    """`nodes` papers without citations, of fitness 1, published in the epoch itself: every weight is 1, the
    first paper is every agent's only anchor and its ball, and one agent cites papers 0, 1, ... in order."""
    n = nodes + 1
    return TraceInput(pub=np.zeros(n, np.int32), fitness=np.ones(n, np.float32), seed_src=np.zeros(0, np.int32),
                      seed_dst=np.zeros(0, np.int32), epoch_nodes=np.array([nodes, n]), epoch_t=np.array([0]),
                      anchors=np.array([[0, -1, -1, -1]], np.int32), cite_off=np.array([0, cites]),
                      cites=np.arange(cites, dtype=np.int32), num_anchors=1)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("nodes,cites", [(3, 2), (3, 3), (40, 30), (1000, 60)])
def test_drawn_weight_above_half_in_64_bits(gpu, nodes, cites, exact):
    """Once more than half of an agent's weight is drawn, log(1 - P / Z) is taken in 64 bits.  Here Z and every P
    are whole numbers and the first citation, of weight beta > nodes, is all that comes before: l = log beta -
    sum_i log D_i, D = Z, then nodes - 1, nodes - 2, ...  Each log is below 12 and good to two ulp (4e-15), twice
    per citation, and every addition rounds a total below 12 per citation."""
    beta = np.random.default_rng(nodes + cites).integers(2 * nodes, 50_000, 40).astype(np.float64)
    pts = np.stack([np.ones(40), np.full(40, 5.0), np.ones(40), beta], axis=1)
    with GrowthEngine(seed=1) as eng:
        eng.set_lik_exact_exp2(exact)
        eng.load_trace(_unit_weight_trace(nodes, cites))
        ll = np.concatenate([eng.loglik(pts), eng.loglik(pts[:7])])
    beta = np.concatenate([beta, beta[:7]])
    left = math.fsum(math.log(nodes - i) for i in range(1, cites))
    want = np.log(beta) - np.log(nodes - 1 + beta) - left
    assert np.abs(ll - want).max() <= cites * (8e-15 + 2.0**-53 * 12 * cites)


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("fitness", [1e38, 1e-30])
def test_weights_at_the_ends_of_the_range(gpu, fitness, exact):
    """A hundred equal weights of 1e38, whose sum is no fp32 number, or of 1e-30: one citation of one of them has
    log-likelihood -log 100, to the fp32 weights' accuracy (1e-7 each in the weight and its logarithm, of which the
    second is relative to 126)."""
    n = 101
    tr = TraceInput(pub=np.zeros(n, np.int32), fitness=np.full(n, fitness, np.float32), seed_src=np.zeros(0, np.int32),
                    seed_dst=np.zeros(0, np.int32), epoch_nodes=np.array([100, n]), epoch_t=np.array([0]),
                    anchors=np.array([[0, -1, -1, -1]], np.int32), cite_off=np.array([0, 1]),
                    cites=np.array([5], np.int32), num_anchors=1)
    pts = np.tile([1.0, 5.0, 1.0, 1.0], (40, 1))
    with GrowthEngine(seed=1) as eng:
        eng.set_lik_exact_exp2(exact)
        eng.load_trace(tr)
        for b in (1, 8, 40):
            assert np.abs(eng.loglik(pts[:b]) + math.log(100.0)).max() <= 2e-5


@pytest.mark.parametrize("points", [3, 20])
def test_weight_table_in_parts_with_balls_in_chunks(gpu, points):
    """Epoch groups of the weight table and chunks of balls that do not end at the same agents: the per-agent
    arithmetic is that of balls kept for all agents, so the results are bitwise equal."""
    g = W.plain_pa_seed(1_100_000, 10, seed=23)
    prm = W.calibration_params()
    prm.growth_rate, prm.fixed_new_nodes = 0.0, 2500
    tr = W.grow_trace(g, prm, 4, seed=7)
    pts = W.theta_batch(points, seed=9)
    with GrowthEngine(seed=1) as a, GrowthEngine(seed=1) as b:
        a.load_trace(tr)
        b.set_tuning(lik_chunk_agents=1700)
        b.load_trace(tr)
        np.testing.assert_array_equal(a.loglik(pts), b.loglik(pts))
        np.testing.assert_array_equal(a.loglik_grad(pts), b.loglik_grad(pts))


@pytest.mark.parametrize("exact", [False, True])
def test_longest_list_drawn_above_half(gpu, exact):
    """256 citations, all but the first from the half of Z that is left, beside others of a short list: the bound of
    test_drawn_weight_above_half_in_64_bits, with logarithms below 15."""
    nodes, cites = 300, 256
    beta = 2.0 ** np.arange(10, 21)
    pts = np.stack([np.ones(11), np.full(11, 5.0), np.ones(11), beta], axis=1)
    pts = np.concatenate([pts] * 4)[:40]
    with GrowthEngine(seed=1) as eng:
        eng.set_lik_exact_exp2(exact)
        eng.load_trace(_unit_weight_trace(nodes, cites))
        ll = np.concatenate([eng.loglik(pts), eng.loglik(pts[:1])])
    b = np.concatenate([pts[:, 3], pts[:1, 3]])
    want = np.log(b) - np.log(nodes - 1 + b) - math.fsum(math.log(nodes - i) for i in range(1, cites))
    assert np.abs(ll - want).max() <= cites * (8e-15 + 2.0**-53 * 15 * cites)
