"""The hot pixels' integer products (csrc/emc_hot.cuh) against the FP64 oracle
and against the gathers alone, at the edges of their tiles.

The plain search leaves the pixels that many frames share to the products;
option tile_skip keeps every photon in the gathers. Both add the same FP32
log-slices (|log W| < 40 here); the gathers' compensated sums round each added
value to 2^-24 of it, the products add exactly.
"""
import numpy as np
import pytest

from common import MODEL_REL_L2, GPUEngine, compare_iteration
from oracle.oracle import EMCProblem, OracleEngine
from dragonfly_b200 import synth

pytestmark = pytest.mark.gpu


def _problem(frames, div, side, photons, zeros=False, big=False, twice=False):
    d = synth.small_problem(seed=frames + div, det_side=side, size=side + 3, qmax=side / 2., n_atoms=60,
                            atom_radius=4., num_div=div, n_frames=frames, mean_count=photons, hole_radius=2.)
    model = d["model_start"] * photons / (d["mask"] == 0).sum() * 2.
    if zeros:   # log 0 inside the detector: some tiles gather all of their photons
        c = model.shape[1] // 2
        model[:, c + 5:c + 8, c:c + 3, c:c + 3] = 0.
    count = d["count_multi"].copy()
    if big:     # counts past a byte keep their pixels out of the products
        count[::97] = 300
        count[5] = 1200
    place = d["place_ones"].copy()
    if twice:   # a pixel listed twice in one frame: both photons count
        mid = (np.cumsum(d["ones"]) - d["ones"] + d["ones"] // 2)[::3]
        place[mid + 1] = place[mid]
    return EMCProblem(d["qvals"], d["corr"], d["mask"], d["ones"], d["multi"], place, d["place_multi"],
                      count, d["quats"], model, need_scaling=1, update_scale=1, beta=0.1)


def _photons(prob):
    n = prob.ones.astype(np.int64).copy()
    np.add.at(n, np.repeat(np.arange(prob.num_data), prob.multi), prob.count_multi)
    return n


@pytest.mark.parametrize("frames,div,side,photons,zeros,big,twice,budget", [
    (256, 1, 24, 150., False, False, False, 0.),    # one row tile exactly, under half an orientation tile
    (257, 2, 24, 200., False, False, False, 0.),    # one frame past it
    (300, 2, 40, 100., False, False, False, 0.),    # some pixels left to the gathers
    (800, 2, 24, 120., False, False, False, 2.0),   # chunks of 267 frames: tomograms added over three
    (511, 1, 24, 200., True, False, False, 0.),     # tiles with log 0
    (400, 2, 24, 250., False, True, False, 0.),     # counts past a byte
    (300, 2, 40, 100., False, False, True, 0.),     # a pixel twice in a frame
])
def test_products_match_oracle_and_gathers(oracle_built, frames, div, side, photons, zeros, big, twice, budget):
    prob = _problem(frames, div, side, photons, zeros, big, twice)
    hot = GPUEngine(prob, pair_budget_mb=budget)
    plain = GPUEngine(prob, pair_budget_mb=budget, tile_skip=1)
    orc = OracleEngine(prob)
    a, b, c = hot.run_iteration(1), orc.run_iteration(1), plain.run_iteration(1)
    assert hot.ctx.workload()["launches"] > plain.ctx.workload()["launches"]   # the products ran
    if budget:
        assert hot.ctx.workload()["chunks"] == 3
    compare_iteration(a, b, prob, 1, model_before=prob.model1)
    np.testing.assert_array_equal(a["rmax"], c["rmax"])
    assert np.all(np.abs(a["likelihood"] - c["likelihood"]) <= 2. ** -24 * 40. * _photons(prob))
    model_before, scale_before = orc.model1(), orc.scale.copy()
    compare_iteration(hot.run_iteration(2), orc.run_iteration(2), prob, 2, model_before=model_before,
                      scale_before=scale_before)
    hot.close()
    plain.close()


@pytest.mark.parametrize("copies,turn,scaling", [
    (2, 1e-9, 1),     # pairs of orientations that only rounding tells apart
    (3, 3e-8, 0),     # the same past it, without scale factors
    (40, 1e-9, 1),    # more near ones than a warp sums at once
    (40, 0., 1),      # exact ties: the lowest index
])
def test_near_ties_fall_as_with_the_gathers(copies, turn, scaling):
    """Every orientation repeated a tiny turn further on: the most likely one of a
    frame and its log-likelihood are the gathers', bit for bit."""
    prob = _problem(300, 1, 24, 200.)
    n = prob.quats.shape[0]
    q = np.repeat(prob.quats, copies, 0)
    q[:, 1:4] += turn * (np.arange(n * copies) % copies)[:, None]
    q[:, :4] /= np.linalg.norm(q[:, :4], axis=1)[:, None]
    q[:, 4] /= copies
    prob = EMCProblem(prob.qvals, prob.corr, prob.mask, prob.ones, prob.multi, prob.place_ones, prob.place_multi,
                      prob.count_multi, q, prob.model1, need_scaling=scaling, update_scale=scaling, beta=0.1)
    got = []
    for skip in (0, 1):
        gpu = GPUEngine(prob, tile_skip=skip)
        got.append(gpu.run_iteration(1))
        assert gpu.ctx.products()["estep"] == 1 - skip
        gpu.close()
    a, b = got
    np.testing.assert_array_equal(a["rmax"], b["rmax"])
    np.testing.assert_array_equal(a["max_exp"], b["max_exp"])


def test_products_lose_no_precision_at_small_logarithms(oracle_built):
    """A start model of about one photon per pixel, where log W is small and FP32
    holds it finely: the digits must too. The gathers' compensated sums round once
    more per photon, so the products' log-likelihoods are as close to the oracle's;
    the model's error is a sum over few orientations here (hence the half)."""
    model, like = [], []
    for seed in (8, 9, 10, 11):
        d, shared = synth.two_detector_problem(seed=seed, n_frames=(300, 200))
        d = d[0]
        prob = EMCProblem(d["qvals"], d["corr"], d["mask"], d["ones"], d["multi"], d["place_ones"], d["place_multi"],
                          d["count_multi"], shared["quats"], shared["model_start"], need_scaling=1, update_scale=1,
                          beta=0.5)
        want = OracleEngine(prob).run_iteration(1)
        off = []
        for skip in (0, 1):
            gpu = GPUEngine(prob, tile_skip=skip)
            got = gpu.run_iteration(1)
            off.append([np.linalg.norm(got[k] - want[k]) for k in ("model1", "likelihood")])
            took = gpu.ctx.products()
            assert took["estep"] == took["mstep"] == 1 - skip and (took["pixels"] >= 128) == (skip == 0)
            gpu.close()
        model.append(off[0][0] / off[1][0])
        like.append(off[0][1] / off[1][1])
    assert model[0] <= 1.5
    assert np.exp(np.mean(np.log(like))) <= 1.


@pytest.mark.parametrize("frames,fits", [(32800, True), (33000, False)])
def test_a_pixel_at_the_range_of_the_accumulators(frames, fits):
    """Every frame has 255 photons on one pixel and is sure of the only orientation: the
    top digits' sum is 250 x 255 x frames, 0.974 of 2^31 at 32800. With 33000 the pixel
    has more than 2^23 photons and stays with the gathers."""
    prob = _problem(300, 1, 24, 200.)
    good = np.nonzero(prob.mask == 0)[0]
    rng = np.random.default_rng(12)
    place = np.concatenate([rng.choice(good[1:], 12, replace=False) for _ in range(frames)]).astype(np.int32)
    ones, multi = np.full(frames, 12, np.int32), np.ones(frames, np.int32)
    prob = EMCProblem(prob.qvals, prob.corr, prob.mask, ones, multi, place, np.full(frames, good[0], np.int32),
                      np.full(frames, 255, np.int32), prob.quats[:1], prob.model1, need_scaling=0, beta=0.1)
    gpu = GPUEngine(prob)
    gpu.ctx.maximize(gpu.ctx.params(1, 0, 0, 0, 1., 100, 1.))
    took = gpu.ctx.products()
    # 512 of the 540 pixels: the bright one and 511 others, or 512 others
    assert took["mstep"] and (took["words"] > 11.9 * frames) == fits
    want = np.bincount(place, minlength=prob.num_pix) / frames
    want[good[0]] = 255.
    np.testing.assert_allclose(gpu.ctx.tomograms(0, 1)[0], want, rtol=4 * 2. ** -24)
    gpu.close()


@pytest.mark.parametrize("cells_per_frame", [0, 1, 6])
def test_tomograms_are_the_sums_over_the_kept_pairs(cells_per_frame):
    """T_r = sum_d P_dr c_d / psum_r from the FP64 probability lists: full search, and
    refined with one cell of seven a frame (most tiles dead, their probability rows --
    here those of a full search before -- not written) and with six (the E-step's
    products too). FP32: P carries three roundings (exp, 1 / norm, product), T one."""
    prob = _problem(300, 2, 24, 200.)
    R, n = prob.quats.shape[0], prob.num_data
    cells = (np.arange(R) * 7 // R).astype(np.int32)         # consecutive orientations share a cell
    rng = np.random.default_rng(3)
    lists = np.array([rng.permutation(7)[:cells_per_frame] for _ in range(n)], np.int32)
    lister, gpu = GPUEngine(prob, keep_prob=1), GPUEngine(prob)
    par = gpu.ctx.params(1, 1, 0, 0, 1., 100, 1.)
    gpu.ctx.maximize(par)
    if cells_per_frame:
        for g in (lister, gpu):
            g.ctx.set_refinement(7, cells, lists)
    lister.ctx.maximize(par)
    gpu.ctx.maximize(par)
    assert gpu.ctx.products()["estep"] and gpu.ctx.products()["mstep"]
    off, place, p = lister.ctx.sparse_prob()
    if cells_per_frame:
        own = np.zeros((n, 7), bool)
        np.put_along_axis(own, lists, True, 1)
        assert np.all(own[np.repeat(np.arange(n), np.diff(off)), cells[place]])
    psum = lister.ctx.orientation_results()[1]
    counts = np.zeros((n, prob.num_pix))
    np.add.at(counts, (np.repeat(np.arange(n), prob.ones), prob.place_ones), 1.)
    np.add.at(counts, (np.repeat(np.arange(n), prob.multi), prob.place_multi), prob.count_multi)
    counts[:, prob.mask > 1] = 0.
    P = np.zeros((R, n))
    P[place, np.repeat(np.arange(n), np.diff(off))] = p
    want = P @ counts
    want[psum > 0] /= psum[psum > 0, None]
    np.testing.assert_allclose(gpu.ctx.tomograms(0, R), want, rtol=4 * 2. ** -24, atol=1e-8 * want.max())
    lister.close()
    gpu.close()


@pytest.mark.parametrize("cells_per_frame,products", [(30, 1), (1, 0)])
def test_refined_estep_on_both_sides_of_its_rule(cells_per_frame, products):
    """A refined search whose frames evaluate many cells takes the E-step's products, one
    with few gathers; both find what the pair lists find, which always gather."""
    prob = _problem(300, 4, 24, 12.)
    R, n = prob.quats.shape[0], prob.num_data
    cells = (np.arange(R) * 108 // R).astype(np.int32)
    rng = np.random.default_rng(4)
    lists = np.array([rng.permutation(108)[:cells_per_frame] for _ in range(n)], np.int32)
    got = []
    for pairs in (0, 1):
        gpu = GPUEngine(prob, pair_lists=pairs)
        gpu.ctx.set_refinement(108, cells, lists)
        gpu.ctx.maximize(gpu.ctx.params(1, 1, 0, 0, 1., 100, 1.))
        took = gpu.ctx.products()
        assert (took["estep"], took["mstep"]) == ((0, 0) if pairs else (products, 1))
        got.append(gpu.ctx.frame_results())
        gpu.close()
    a, b = got
    np.testing.assert_array_equal(a["rmax"], b["rmax"])
    assert np.all(np.abs(a["likelihood"] - b["likelihood"]) <= 2. ** -24 * 40. * _photons(prob))


def test_tiles_that_gather_all_take_no_products():
    """One of two modes is empty: each tile has log 0, gathers all of its photons and its
    products are left out. A withheld stage that only E-step products would reach (their
    depth is the pixels, the M-step's the 256 frames) shows that none ran."""
    prob = _problem(256, 2, 40, 600.)
    model = np.concatenate([prob.model1, 0. * prob.model1])
    prob = EMCProblem(prob.qvals, prob.corr, prob.mask, prob.ones, prob.multi, prob.place_ones, prob.place_multi,
                      prob.count_multi, prob.quats, model, need_scaling=1, update_scale=1, beta=0.1)
    assert prob.num_modes == 2
    got = []
    for skip in (0, 1):
        gpu = GPUEngine(prob, tile_skip=skip, dense_wait_cycles=2e7, dense_withhold_stage=3)
        got.append(gpu.run_iteration(1))
        took = gpu.ctx.products()
        assert took["estep"] == 1 - skip and (took["pixels"] > 3 * 128) == (skip == 0)
        gpu.close()
    a, b = got
    np.testing.assert_array_equal(a["rmax"], b["rmax"])
    np.testing.assert_array_equal(a["max_exp"], b["max_exp"])
    assert np.all(a["rmax"] % 2 == 0)


def test_more_tiles_than_a_grid_extent_of_their_halves():
    """32768 orientation tiles (4.2 million orientations): twice as many 64-orientation
    halves as a grid's second extent takes. The products find what the gathers find."""
    prob = _problem(256, 1, 24, 200.)
    rng = np.random.default_rng(9)
    q = rng.normal(size=(32768 * 128, 5))
    q[:, :4] /= np.linalg.norm(q[:, :4], axis=1)[:, None]
    q[:, 4] = 1. / q.shape[0]
    got = []
    for skip in (0, 1):
        gpu = GPUEngine(prob, tile_skip=skip, pair_budget_mb=30000)
        gpu.ctx.set_quaternions(q)
        gpu.ctx.maximize(gpu.ctx.params(1, 1, 0, 0, 1., 100, 1.))
        assert gpu.ctx.products()["estep"] == gpu.ctx.products()["mstep"] == 1 - skip
        gpu.ctx.update_model(0.)
        got.append((gpu.ctx.frame_results(), gpu.ctx.model()[0]))
        gpu.close()
    (a, ma), (b, mb) = got
    np.testing.assert_array_equal(a["rmax"], b["rmax"])
    assert np.all(np.abs(a["likelihood"] - b["likelihood"]) <= 2. ** -24 * 40. * _photons(prob))
    assert np.linalg.norm(ma - mb) <= MODEL_REL_L2 * np.linalg.norm(mb)


@pytest.mark.parametrize("refused", [1, 2, 3])
def test_without_memory_for_the_products(refused):
    """No memory for the log-slices' digits: the E-step gathers and the M-step keeps its
    products; none for the counts: both gather. The same later, when more orientations
    need larger buffers than the first call's."""
    small, large = _problem(300, 1, 24, 200.), _problem(300, 2, 24, 200.)
    plain, gpu = GPUEngine(small, tile_skip=1), GPUEngine(small)
    par = plain.ctx.params(1, 1, 0, 0, 1., 100, 1.)
    c = gpu.ctx
    for first in (True, False):
        if not first:
            for g in (plain, gpu):
                g.ctx.set_quaternions(large.quats)
        for mem in (0, refused) if first else (refused, 0):
            c.set_option("refuse_memory", mem)
            for g in (plain, gpu):
                g.ctx.maximize(par)
            took = c.products()
            assert (took["estep"], took["mstep"]) == (int(mem == 0), int(mem < 2))
            a, b = c.frame_results(), plain.ctx.frame_results()
            np.testing.assert_array_equal(a["rmax"], b["rmax"])
            assert np.all(np.abs(a["likelihood"] - b["likelihood"]) <= 2. ** -24 * 40. * _photons(small))
            want = plain.ctx.tomograms(0, 60)
            np.testing.assert_allclose(c.tomograms(0, 60), want, rtol=8 * 2. ** -24, atol=1e-8 * want.max())
    plain.close()
    gpu.close()


def test_products_give_their_memory_back():
    """A context that goes from a full search to pair lists holds no more than one that
    began with them (the count matrices alone are 20 MB here)."""
    import torch
    prob = _problem(300, 2, 24, 200.)
    n, R = 20100, prob.quats.shape[0]
    rep = lambda a: np.tile(a, n // 300)
    prob = EMCProblem(prob.qvals, prob.corr, prob.mask, rep(prob.ones), rep(prob.multi), rep(prob.place_ones),
                      rep(prob.place_multi), rep(prob.count_multi), prob.quats, prob.model1, need_scaling=1,
                      update_scale=1, beta=0.1)
    cells = (np.arange(R) * 7 // R).astype(np.int32)
    lists = np.tile(np.array([[0, 3]], np.int32), (n, 1))
    held = []
    for full_first in (False, True):
        before = torch.cuda.mem_get_info()[0]
        gpu = GPUEngine(prob)
        par = gpu.ctx.params(1, 1, 0, 0, 1., 100, 1.)
        if full_first:
            gpu.ctx.maximize(par)
            assert gpu.ctx.products()["pixels"] >= 256
        gpu.ctx.set_refinement(7, cells, lists)
        gpu.ctx.set_option("pair_lists", 1)
        gpu.ctx.set_option("block_budget_mb", 16)
        gpu.ctx.maximize(par)
        assert gpu.ctx.products()["pixels"] == 0
        held.append(before - torch.cuda.mem_get_info()[0])
        gpu.close()
    assert held[1] - held[0] <= 8 << 20


def test_product_wait_gives_up_and_the_context_recovers(oracle_built):
    """A stage whose copies are withheld (test hook): its waits run out, the
    kernels return, the call reports the error, and the next call succeeds."""
    from dragonfly_b200._lib import DFG_ERR_CUDA, DFGError
    prob = _problem(257, 2, 24, 200.)
    gpu = GPUEngine(prob)
    c = gpu.ctx
    par = c.params(1, 1, 1, 0, 1., 100, 1.)
    c.set_option("dense_wait_cycles", 2e7)
    c.set_option("dense_withhold_stage", 1)
    with pytest.raises(DFGError) as e:
        c.maximize(par)
    assert e.value.code == DFG_ERR_CUDA and "gave up" in str(e.value)
    c.set_option("dense_withhold_stage", -1)
    c.set_option("dense_wait_cycles", 2e9)
    c.set_scale(np.ones(prob.num_data))   # the failed call's scale update is invalid with its other results
    a = gpu.run_iteration(1)
    compare_iteration(a, OracleEngine(prob).run_iteration(1), prob, 1, model_before=prob.model1)
    gpu.close()
