"""Parity of the CUDA path (libdfgpu.so through its C ABI) with the FP64 oracle.

Bar (the plain form against the reference engine with one-thread semantics):
model relative L2 <= 1e-5 after every iteration, average log-likelihood and
mutual information within 1e-6 relative, the same most likely orientation for
>= 99.9 % of frames, scale factors within 1e-5 relative.
"""
import numpy as np
import pytest

from common import (CASES, GPUEngine, compare_iteration, load_case, rel_l2)
from dragonfly_b200._lib import Context
from oracle.oracle import EMCProblem, OracleEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", CASES)
def test_gpu_matches_oracle_on_golden_cases(name, oracle_built):
    prob, g = load_case(name)
    gpu = GPUEngine(prob)
    orc = OracleEngine(prob)
    for it in range(1, int(g["iters"]) + 1):
        model_before, scale_before = orc.model1(), orc.scale.copy()
        a = gpu.run_iteration(it)
        b = orc.run_iteration(it)
        dev = compare_iteration(a, b, prob, it, model_before=model_before, scale_before=scale_before)
        # the golden vectors of the reference itself
        k = "it%d_" % it
        good = g["blacklist"] == 0
        assert np.mean(a["rmax"][good] == g[k + "rmax"][good]) >= 0.999 - dev["rmax_ties"] / good.sum()
        assert np.all(a["rmax"][~good] == -1)
        assert abs(a["avg_likelihood"] - g[k + "scalars"][0]) <= 1e-6 * abs(g[k + "scalars"][0])
        # u_r and the rescale factor are FP64 sums in the reference's order:
        # bit-identical on the shared start model; afterwards the models differ
        # within the model tolerance
        if it == 1:
            np.testing.assert_array_equal(a["u"], b["u"])
            assert a["rescale"] == b["rescale"]
        else:
            np.testing.assert_allclose(a["u"], b["u"], rtol=1e-6)
            assert abs(a["rescale"] - b["rescale"]) <= 1e-6 * abs(b["rescale"])
        # kept-set sizes: the pruning rule of max_prob.c:184-203
        assert np.mean(a["num_prob"] == b["num_prob"]) >= 0.999
        if prob.num_modes > 1:
            np.testing.assert_allclose(a["quat_norm"], b["quat_norm"], rtol=1e-5, atol=1e-9)
    assert rel_l2(a["model1"], g["final_model1"]) <= 1e-5
    gpu.close()


def test_gpu_small_config_ten_iterations(oracle_built):
    """The small CPU-runnable configuration: 64x64 detector, 75^3 model,
    3240 orientations, 3000 frames at 50 photons, beta = 1, 10 iterations."""
    from dragonfly_b200 import synth
    d = synth.small_problem(seed=0)
    prob = EMCProblem(d["qvals"], d["corr"], d["mask"], d["ones"], d["multi"], d["place_ones"],
                      d["place_multi"], d["count_multi"], d["quats"], d["model_start"], beta=1.)
    gpu = GPUEngine(prob)
    orc = OracleEngine(prob)
    worst = {}
    for it in range(1, 11):
        model_before = orc.model1()
        a = gpu.run_iteration(it)
        b = orc.run_iteration(it)
        dev = compare_iteration(a, b, prob, it, model_before=model_before)
        for k, v in dev.items():
            if isinstance(v, float):
                worst[k] = max(worst.get(k, 0.), v) if k != "rmax_agree" else min(worst.get(k, 1.), v)
    print("small config worst deviations over 10 iterations:", worst)
    gpu.close()


def test_gpu_frame_chunks_agree(oracle_built):
    """Splitting the frames into chunks (bounded per-pair memory) gives the same
    iteration as one chunk."""
    prob, _ = load_case("scaling")
    one = GPUEngine(prob)
    many = GPUEngine(prob, pair_budget_mb=0.05)
    for it in (1, 2):
        a = one.run_iteration(it)
        b = many.run_iteration(it)
        assert many.ctx.workload()["chunks"] > 1
        assert rel_l2(a["model1"], b["model1"]) <= 1e-6
        np.testing.assert_array_equal(a["rmax"], b["rmax"])
        assert abs(a["avg_likelihood"] - b["avg_likelihood"]) <= 1e-9 * abs(b["avg_likelihood"])
    one.close()
    many.close()


@pytest.mark.parametrize("case", ["scaling", "beta1"])
def test_gpu_orientation_blocks_agree(oracle_built, case):
    """The orientation-blocked two-pass full search (block_budget_mb: a few
    tiles of log-slices and tomograms at a time; the E-step done twice, the
    second pass forming the probabilities from the first pass's per-frame
    maximum, first argmax and kept sum) gives the iteration of the resident
    layout with the same frame chunks: the same log-likelihood sums, kept
    pairs and probabilities, tomograms summed in the same chunk order (the
    merge's FP64 atomics differ in order only)."""
    prob, _ = load_case(case)
    many = GPUEngine(prob, pair_budget_mb=0.05, keep_prob=1)
    blk = GPUEngine(prob, pair_budget_mb=0.05, block_budget_mb=1.1, keep_prob=1)   # one tile per block
    for it in (1, 2):
        a = many.run_iteration(it)
        b = blk.run_iteration(it)
        assert blk.ctx.workload()["chunks"] > 1
        assert rel_l2(a["model1"], b["model1"]) <= 1e-10, rel_l2(a["model1"], b["model1"])
        np.testing.assert_array_equal(a["rmax"], b["rmax"])
        np.testing.assert_allclose(a["likelihood"], b["likelihood"], rtol=1e-13, atol=1e-13)
        # psum_r sums the stored FP32 probabilities (E = exp(beta (x - max))
        # rounded to FP32, then times 1 / p_norm in FP32): a log-likelihood
        # one bit apart between the two E-step layouts can move one of them by
        # an FP32 ulp
        np.testing.assert_allclose(a["psum_r"], b["psum_r"], rtol=1e-9, atol=1e-300)
        oa, pa, va = many.ctx.sparse_prob()
        ob, pb, vb = blk.ctx.sparse_prob()
        np.testing.assert_array_equal(oa, ob)
        np.testing.assert_array_equal(pa, pb)
        # after the first merge the models differ in the last bits (FP64
        # atomics in another order), and the probabilities by about 1e-15
        np.testing.assert_allclose(va, vb, rtol=1e-12, atol=0.)
    with pytest.raises(RuntimeError):
        blk.ctx.tomograms(0, 1)        # one block of tomograms at a time
    many.close()
    blk.close()


def test_gpu_is_deterministic(oracle_built):
    prob, _ = load_case("beta1")
    a = GPUEngine(prob).run_iteration(1)
    b = GPUEngine(prob).run_iteration(1)
    np.testing.assert_array_equal(a["rmax"], b["rmax"])
    np.testing.assert_array_equal(a["likelihood"], b["likelihood"])
    np.testing.assert_array_equal(a["p_norm"], b["p_norm"])


def test_gpu_context_reused_for_another_detector():
    """A context whose log-slices have room from a small detector with many orientations
    goes to a larger one, first with few orientations, then with more: what it finds is
    what a new context finds."""
    from dragonfly_b200 import synth
    from dragonfly_b200.quatgen import quat_gen

    def load(c, d, div):
        c.set_detector(d["qvals"], d["corr"], d["mask"])
        c.set_frames(d["ones"], d["multi"], d["place_ones"], d["place_multi"], d["count_multi"])
        c.set_quaternions(quat_gen(div))
        c.set_model(d["model_start"])
        c.calc_beta(0.1, 0)
        c.maximize(c.params(1, 0, 0, 0, 1., 100, 1.))
        return c.frame_results()

    small, large = (synth.small_problem(seed=side, det_side=side, size=side + 3, qmax=side / 2., n_atoms=40,
                                        atom_radius=4., num_div=1, n_frames=200, mean_count=60., hole_radius=2.)
                    for side in (24, 40))
    used = Context(0)
    load(used, small, 4)
    for div in (1, 2, 3):
        new = Context(0)
        a, b = load(used, large, div), load(new, large, div)
        for k in ("rmax", "likelihood", "max_exp"):
            np.testing.assert_array_equal(a[k], b[k])
        new.close()
    used.close()


def test_gpu_frames_beyond_a_new_detector_are_dropped():
    """A smaller detector under frames that list pixels past it is refused, and the frames
    with it: an iteration wants them set again."""
    from dragonfly_b200 import synth
    from dragonfly_b200._lib import DFG_ERR_ARG, DFG_ERR_STATE, DFGError
    from dragonfly_b200.quatgen import quat_gen
    small, large = (synth.small_problem(seed=side, det_side=side, size=side + 3, qmax=side / 2., n_atoms=40,
                                        atom_radius=4., num_div=1, n_frames=50, mean_count=60., hole_radius=2.)
                    for side in (24, 40))
    c = Context(0)

    def frames(d):
        c.set_frames(d["ones"], d["multi"], d["place_ones"], d["place_multi"], d["count_multi"])

    c.set_detector(large["qvals"], large["corr"], large["mask"])
    frames(large)
    c.set_quaternions(quat_gen(1))
    c.set_model(small["model_start"])
    c.calc_beta(0.1, 0)
    par = c.params(1, 0, 0, 0, 1., 100, 1.)
    c.maximize(par)
    with pytest.raises(DFGError) as e:
        c.set_detector(small["qvals"], small["corr"], small["mask"])
    assert e.value.code == DFG_ERR_ARG
    with pytest.raises(DFGError) as e:
        c.maximize(par)
    assert e.value.code == DFG_ERR_STATE
    c.set_detector(small["qvals"], small["corr"], small["mask"])
    frames(small)
    c.calc_beta(0.1, 0)
    c.maximize(par)
    assert np.all(np.isfinite(c.frame_results()["likelihood"]))
    c.close()


def test_gpu_slice_gen_and_merge_match_oracle(oracle_built):
    import ctypes as C
    prob, _ = load_case("beta1")
    gpu = GPUEngine(prob)
    orc = OracleEngine(prob)
    for r in (0, 33, 211, 419):
        a = gpu.ctx.slice_gen(prob.quats[r])
        b = orc.slice_gen(prob.quats[r])
        np.testing.assert_array_equal(a, b)  # FP64 geometry in the reference's operation order
    # merge one view into zeroed host grids
    view = orc.slice_gen(prob.quats[5])
    m2 = np.zeros(prob.model1.shape)
    w = np.zeros(prob.model1.shape)
    gpu.ctx.slice_merge(prob.quats[5], view, m2, w)
    m2o = np.zeros(prob.model1.shape)
    wo = np.zeros(prob.model1.shape)
    orc.lib.orc_slice_merge3d(np.ascontiguousarray(prob.quats[5]), 0, view, m2o.reshape(-1), wo.reshape(-1),
                              prob.size, prob.num_pix, prob.qvals.reshape(-1), prob.corr, prob.mask)
    np.testing.assert_allclose(m2, m2o, rtol=1e-12, atol=1e-15)
    np.testing.assert_allclose(w, wo, rtol=1e-12, atol=1e-15)
    gpu.close()


def test_gpu_rejects_bad_inputs():
    from dragonfly_b200._lib import Context, DFGError
    prob, _ = load_case("beta1")
    c = Context(0)
    with pytest.raises(DFGError):  # frames before detector
        c.set_frames(prob.ones, prob.multi, prob.place_ones, prob.place_multi, prob.count_multi)
    c.set_detector(prob.qvals, prob.corr, prob.mask)
    bad = prob.place_ones.copy()
    bad[3] = prob.num_pix + 5
    with pytest.raises(DFGError, match="out of"):
        c.set_frames(prob.ones, prob.multi, bad, prob.place_multi, prob.count_multi)
    q = prob.quats.copy()
    q[2, 1] = np.nan
    with pytest.raises(DFGError, match="not finite"):
        c.set_quaternions(q)
    with pytest.raises(DFGError):  # iteration before inputs
        c.maximize(c.params(1))
    c.close()
