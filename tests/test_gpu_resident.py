"""The one-launch path for windows whose rows fit on the chip, at the sizes where its partition changes: one row, the
last row of a 32-row unit and of a CTA, one cluster full and one row more, the largest window (on a GPU that holds 15
clusters of eight CTAs) and one row more (one launch per step again), and window counts that take clusters of 8, 4, 2 and 1
CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 961
TOL = {0: 1e-5, 1: 2e-3}


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("W,rows", [(1, 1), (1, 33), (1, 4096), (1, 4097), (1, 61440), (1, 61441), (3, 9001), (15, 300),
                                    (16, 2048), (40, 1000), (100, 511)])
def test_resident_launch_matches_oracle_and_per_step_launches(built, monkeypatch, prec, W, rows):
    m, O = built
    n_iter, L = 4, 3
    cfg = m.reference_config(precision=prec, leapfrog_steps=L, burn_in=1, adapt_steps=3, sample_capacity=n_iter,
                             trace_iters=n_iter, seed=5, eps0=0.02)
    data = [m.synth_window(31, g, rows) for g in range(min(W, 3))]
    w = (0.15 * np.random.default_rng(rows).standard_normal(P)).astype(np.float32)
    mom = np.random.default_rng(1).standard_normal(P).astype(np.float32)

    def run():
        ctx = m.Context(cfg, n_windows=W, rows=rows)
        for i in range(W):
            x, y, _ = data[i % len(data)]
            ctx.set_window_data(i, x, y, global_window=i)
        grad = ctx.potential_and_grad(W - 1, w, want_row_loss=True)
        steps = ctx.leapfrog(W - 1, 4, 1e-3, w, mom, grad["grad"])
        ctx.run_chain(1)
        ctx.run_chain(n_iter - 1)
        out = [(ctx.get_samples(i), ctx.get_trace(i), ctx.chain_info(i), ctx.get_state(i)) for i in (0, W - 1)]
        n = ctx.launch_count(), ctx.resident_plan(), ctx.resident_plan(explicit_calls=True)
        ctx.close()
        return grad, steps, out, n

    grad, steps, chains, (n_one, plan, plan_x) = run()
    monkeypatch.setenv("MCMC_B200_NO_MULTISTEP", "1")
    grad_s, steps_s, chains_s, (n_many, none, none_x) = run()
    assert none == none_x == (0, 0)
    assert (n_one < n_many) == (plan[0] > 0 or plan_x[0] > 0)
    for c, k in (plan, plan_x):
        assert c * k * 512 >= rows or c == 0
    assert rows <= 61440 or plan_x == (0, 0)
    assert rows > 4096 or plan_x == (8, 1)
    x, y, _ = data[(W - 1) % len(data)]
    ref = O.logp_grad(O.reference_model(tf32=bool(prec)), x, y, w, want_losses=True)
    tol = TOL[prec]
    for got in (grad, grad_s):
        assert np.abs(got["grad"] - ref["grad"]).max() <= tol * np.abs(ref["grad"]).max()
        assert abs(got["loglik"] - ref["loglik"]) <= tol * abs(ref["loglik"])
        assert abs(got["logprior"] - ref["logprior"]) <= 1e-6 * abs(ref["logprior"])
        assert np.allclose(got["row_loss"], ref["row_loss"], rtol=10 * tol, atol=10 * tol)
    # the two paths add the same rows in another order
    for k in ("w_next", "mom_next", "grad_cur"):
        assert np.abs(steps[k] - steps_s[k]).max() <= 1e-4 * np.abs(steps_s[k]).max(), k
    for (s1, t1, i1, g1), (s2, t2, i2, g2) in zip(chains, chains_s):
        assert i1 == i2 and np.array_equal(t1["accepted"], t2["accepted"])
        assert np.array_equal(t1["momenta"], t2["momenta"]) and np.array_equal(t1["log_u"], t2["log_u"])
        assert np.array_equal(t1["eps"], t2["eps"])
        assert np.allclose(t1["log_acpt"], t2["log_acpt"], rtol=1e-3, atol=1e-3)
        assert np.abs(s1[:n_iter - 1] - s2[:n_iter - 1]).max() <= 1e-4 * max(1e-3, np.abs(s2[:n_iter - 1]).max())
        assert abs(g1["loglik"] - g2["loglik"]) <= 1e-6 * abs(g2["loglik"])


@pytest.mark.parametrize("W,rows,clusters", [(1, 2560, 1), (1, 2561, 3), (4, 3584, 1), (4, 3585, 3), (7, 4096, 2), (8, 4096, 1)])
def test_fp32_chains_on_several_clusters_below_one_clusters_rows(built, monkeypatch, W, rows, clusters):
    """Where a chain's window is dealt to several clusters although one would hold it; explicit calls keep one.  Results as above."""
    m, _ = built
    ctx = m.Context(m.reference_config(precision=0, sample_capacity=0), n_windows=W, rows=rows)
    assert ctx.resident_plan() == (8, clusters) and ctx.resident_plan(explicit_calls=True) == (8, 1)
    ctx.close()
    test_resident_launch_matches_oracle_and_per_step_launches(built, monkeypatch, 0, W, rows)


@pytest.mark.parametrize("rows", [1025, 2049, 4096, 16500, 30000, 61440])
def test_fp32_steps_and_evaluations_agree(built, rows):
    """Steps go by integers, evaluations on host pointers by FFMA: the gradient that a step ends with is the evaluation's at its end, and three
    steps are three times one, but for FP32 rounding, 1e-5 of the largest as against the oracle."""
    m, _ = built
    x, y, _ = m.synth_window(7, 0, rows)
    ctx = m.Context(m.reference_config(precision=0, sample_capacity=0), 1, rows)
    ctx.set_window_data(0, x, y)
    rng = np.random.default_rng(rows)
    w, mom = (0.15 * rng.standard_normal(P)).astype(np.float32), rng.standard_normal(P).astype(np.float32)
    start = ctx.potential_and_grad(0, w)["grad"]
    whole = ctx.leapfrog(0, 3, 1e-4, w, mom, start)
    g = start
    for _ in range(3):
        s = ctx.leapfrog(0, 1, 1e-4, w, mom, g)
        w, mom, g = s["w_next"], s["mom_next"], s["grad_cur"]
        assert np.abs(g - ctx.potential_and_grad(0, w)["grad"]).max() <= 1e-5 * np.abs(g).max()
    for k, v in (("w_next", w), ("grad_cur", g)):
        assert np.abs(whole[k] - v).max() <= 1e-5 * np.abs(v).max()
    ctx.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_a_wait_that_runs_out_reports_and_leaves_the_chain_where_it_was(built, prec):
    """One cluster of the window is left out of a launch, so that the others' waits for its words run out: by themselves,
    with a status, and without a step of the chain."""
    m, _ = built
    rows = 9001
    x, y, _ = m.synth_window(8, 0, rows)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)

    def run(disturbed):
        ctx = m.Context(m.reference_config(precision=prec, leapfrog_steps=3, burn_in=0, sample_capacity=8, seed=3), 1, rows)
        ctx.set_window_data(0, x, y)
        if disturbed:
            code, msg = ctx.selftest_resident_wait(603)
            assert code == 4 and "603" in msg, (code, msg)
        out = [ctx.potential_and_grad(0, w)["grad"]]
        ctx.run_chain(4)
        if disturbed:
            before = ctx.get_state(0), ctx.chain_info(0)
            code, msg = ctx.selftest_resident_wait(603)
            assert code == 4 and "603" in msg, (code, msg)
            after = ctx.get_state(0), ctx.chain_info(0)
            assert before[1] == after[1] and all(np.array_equal(before[0][k], after[0][k]) for k in before[0])
            ctx.synchronize()  # reported once
        ctx.run_chain(4)
        out += [ctx.get_samples(0), ctx.potential_and_grad(0, w)["grad"]]
        ctx.close()
        return out

    for a, b in zip(run(True), run(False)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("code", [611, 901])
def test_evaluations_report_rows_that_do_not_arrive_and_earlier_time_outs(built, prec, code):
    m, _ = built
    x, y, _ = m.synth_window(8, 0, 700)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)
    ctx = m.Context(m.baseline_config(precision=prec), 1, 700)
    ctx.set_window_data(0, x, y)
    before = ctx.potential_and_grad(0, w)
    got, msg = ctx.selftest_resident_wait(code)
    assert got == 4 and str(code) in msg, (got, msg)
    after = ctx.potential_and_grad(0, w)
    assert np.array_equal(before["grad"], after["grad"]) and before["loglik"] == after["loglik"]
    ctx.close()


@pytest.mark.parametrize("rows", [700, 58368])
@pytest.mark.parametrize("code", [612, 613])
def test_evaluations_report_products_that_do_not_end(built, code, rows):
    m, _ = built
    x, y, _ = m.synth_window(8, 0, rows)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)
    ctx = m.Context(m.baseline_config(precision=m.PREC_FP32), 1, rows)
    ctx.set_window_data(0, x, y)
    before = ctx.potential_and_grad(0, w)
    got, msg = ctx.selftest_resident_wait(code)
    assert got == 4 and str(code) in msg, (got, msg)
    after = ctx.potential_and_grad(0, w)
    assert np.array_equal(before["grad"], after["grad"]) and before["loglik"] == after["loglik"]
    ctx.close()


@pytest.mark.parametrize("prec,most", [(0, 10000), (1, 20000)])
def test_trajectories_above_a_launch_of_a_tenth_of_a_second_take_one_launch_per_step(built, prec, most):
    m, _ = built
    x, y, _ = m.synth_window(8, 0, 64)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)
    for L, per_step in ((most, False), (most + 1, True)):
        ctx = m.Context(m.reference_config(precision=prec, leapfrog_steps=L, burn_in=0, adapt_steps=0, sample_capacity=1,
                                           eps0=1e-6), 1, 64)
        ctx.set_window_data(0, x, y)
        ctx.launch_count(reset=True)
        out = ctx.leapfrog(0, L, 1e-6, w, w, w)
        assert (ctx.launch_count(reset=True) > L) == per_step and np.isfinite(out["w_next"]).all()
        ctx.run_chain(1)
        assert (ctx.launch_count() > L) == per_step and ctx.chain_info(0)["iterations"] == 1
        ctx.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_a_refused_launch_becomes_one_launch_per_step(built, monkeypatch, prec):
    """The driver's answer to a launch that does not fit is made on the host."""
    import torch
    m, _ = built
    rows, L = 5000, 3
    x, y, _ = m.synth_window(8, 0, rows)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)
    xd, yd, wd = (torch.from_numpy(v).cuda() for v in (x, y, w))

    def run(refuse):
        ctx = m.Context(m.reference_config(precision=prec, leapfrog_steps=L, burn_in=0, sample_capacity=6), 1, rows)
        ctx.set_window_data(0, x, y)
        out = []
        if refuse:
            ctx.selftest_refuse_resident(1)
        out.append(ctx.potential_and_grad(0, w, want_row_loss=True)["row_loss"])
        if refuse:
            ctx.selftest_refuse_resident(1)
        out.append(ctx.leapfrog(0, L, 1e-3, w, w, w)["w_next"])
        if refuse:
            ctx.selftest_refuse_resident(1)
        ctx.run_chain(6)
        out.append(ctx.get_samples(0))
        b = [torch.full((P,), 7.0, device="cuda") for _ in range(4)]
        loss = torch.zeros(rows + P, device="cuda")
        torch.cuda.synchronize()
        if refuse:
            ctx.selftest_refuse_resident(1)
        ctx.mcmc_step(xd.data_ptr(), yd.data_ptr(), wd.data_ptr(), b[0].data_ptr(), wd.data_ptr(), b[1].data_ptr(),
                      wd.data_ptr(), b[2].data_ptr(), b[3].data_ptr(), loss.data_ptr(), L, 1e-3)
        ctx.synchronize()
        out += [v.cpu().numpy() for v in b] + [loss.cpu().numpy()]
        n = ctx.launch_count()
        ctx.close()
        return out, n

    monkeypatch.delenv("MCMC_B200_NO_MULTISTEP", raising=False)
    refused, n_refused = run(True)
    monkeypatch.setenv("MCMC_B200_NO_MULTISTEP", "1")
    per_step, n_per_step = run(False)
    assert n_refused == n_per_step
    for a, b in zip(refused, per_step):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [0, 1])
def test_reference_random_streams_on_the_chip(built, monkeypatch, prec):
    m, _ = built
    rows, n_iter = 5000, 6
    x, y, _ = m.synth_window(8, 0, rows)

    def run():
        cfg = m.reference_config(precision=prec, leapfrog_steps=3, burn_in=1, adapt_steps=4, sample_capacity=n_iter,
                                 trace_iters=n_iter, seed=11, eps0=0.02, rng_streams=m.RNG_REFERENCE)
        ctx = m.Context(cfg, 1, rows)
        ctx.set_window_data(0, x, y)
        plan = ctx.resident_plan()
        ctx.run_chain(2)          # (the host's accept draws are extended between launches)
        ctx.run_chain(n_iter - 2)
        out = ctx.get_samples(0)[:n_iter - 1], ctx.get_trace(0), ctx.chain_info(0)
        ctx.close()
        return plan, out

    plan, (s1, t1, i1) = run()
    monkeypatch.setenv("MCMC_B200_NO_MULTISTEP", "1")
    none, (s2, t2, i2) = run()
    assert plan != (0, 0) and none == (0, 0)
    assert i1 == i2 and np.array_equal(t1["momenta"], t2["momenta"]) and np.array_equal(t1["log_u"], t2["log_u"])
    assert np.array_equal(t1["accepted"], t2["accepted"]) and np.array_equal(t1["eps"], t2["eps"])
    assert np.abs(s1 - s2).max() <= 1e-4 * max(1e-3, np.abs(s2).max())


@pytest.mark.parametrize("prec", [0, 1])
def test_a_diverging_trajectory_rejects_and_the_chain_stays(built, monkeypatch, prec):
    """Steps so long that weights become infinite and NaN: what travels with the weights then is no report of a wait."""
    m, _ = built
    rows = 5000
    x, y, _ = m.synth_window(8, 0, rows)

    def run(eps0):
        ctx = m.Context(m.baseline_config(precision=prec, leapfrog_steps=8, sample_capacity=4, trace_iters=4, eps0=eps0), 1, rows)
        ctx.set_window_data(0, x, y)
        ctx.run_chain(4)
        out = ctx.get_samples(0), ctx.get_trace(0)["accepted"], ctx.chain_info(0), ctx.get_state(0)
        ctx.close()
        return out

    for eps0 in (1e19, 1e30):
        monkeypatch.delenv("MCMC_B200_NO_MULTISTEP", raising=False)
        s1, a1, i1, g1 = run(eps0)
        monkeypatch.setenv("MCMC_B200_NO_MULTISTEP", "1")
        s2, a2, i2, g2 = run(eps0)
        assert not a1.any() and not a2.any() and i1 == i2
        assert not s1.any() and not s2.any()   # the chain's start, w = 0
        # (the start's gradient is the bootstrap launch's in both)
        assert np.array_equal(g1["grad"], g2["grad"]) and g1["loglik"] == g2["loglik"]


def _step_args(m, torch, ctx, x, y, in_place):
    P_ = ctx.P
    g = torch.Generator(device="cuda").manual_seed(4)
    w, mom, grad = (0.1 * torch.randn(P_, device="cuda", generator=g) for _ in range(3))
    out = [w, mom, grad] if in_place else [torch.zeros(P_, device="cuda") for _ in range(3)]
    zero, loss = torch.ones(P_, device="cuda"), torch.zeros(x.shape[0] + P_, device="cuda")
    torch.cuda.synchronize()
    keep = (w, mom, grad, zero, loss)
    p = [t.data_ptr() for t in (x, y, w, out[0], mom, out[1], grad, out[2], zero, loss)]
    return p, out + [zero, loss], keep


@pytest.mark.parametrize("prec", [0, 1])
def test_mcmc_step_in_place_and_replayed_from_a_graph(built, prec):
    import torch
    m, _ = built
    rows, L = 9001, 4
    ctx = m.Context(m.reference_config(precision=prec, sample_capacity=0), 1, rows)
    x, y = (torch.from_numpy(v).cuda() for v in m.synth_window(8, 0, rows)[:2])
    res = {}
    for in_place in (False, True):
        p, out, keep = _step_args(m, torch, ctx, x, y, in_place)
        ctx.mcmc_step(*p, L, 1e-3)
        ctx.synchronize()
        res[in_place] = [v.cpu().numpy() for v in out]
    assert not res[False][3].any()     # grad_next
    for a, b in zip(res[False], res[True]):
        assert np.array_equal(a, b)
    # captured once, replayed three times
    p, out, keep = _step_args(m, torch, ctx, x, y, False)
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.mcmc_step(*p, L, 1e-3, stream=s.cuda_stream)
    for _ in range(3):
        for v in out:
            v.fill_(5.0)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, res[False]):
            assert np.array_equal(a.cpu().numpy(), b)
    del graph
    ctx.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_two_contexts_at_once(built, prec):
    """Two chains of 120 CTAs each, from two threads on their own streams: neither launch may hold SMs while it waits for
    the other's."""
    import threading
    m, _ = built
    rows, n = 58368, 40
    data = m.synth_window(8, 0, rows)[:2]

    def make():
        ctx = m.Context(m.reference_config(precision=prec, leapfrog_steps=5, burn_in=0, adapt_steps=0, sample_capacity=n,
                                           seed=1), 1, rows)
        ctx.set_window_data(0, *data)
        return ctx

    alone = make()
    alone.run_chain(n)
    want = alone.get_samples(0)
    alone.close()
    both, errors = [make(), make()], []

    def work(ctx):
        try:
            for _ in range(n // 2):
                ctx.run_chain(2)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in both]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for c in both:
        assert np.array_equal(c.get_samples(0), want)
        c.close()


@pytest.mark.parametrize("rows", [1025, 4096, 16500, 58368])
@pytest.mark.parametrize("code", [621, 622, 623, 624])
def test_steps_by_integers_report_waits_that_run_out(built, code, rows):
    """The tile arithmetic of FP32 steps (evaluations have another): 611 to 614 in it."""
    m, _ = built
    x, y, _ = m.synth_window(8, 0, rows)
    w = (0.1 * np.random.default_rng(2).standard_normal(P)).astype(np.float32)
    ctx = m.Context(m.baseline_config(precision=m.PREC_FP32), 1, rows)
    ctx.set_window_data(0, x, y)
    before = ctx.leapfrog(0, 3, 1e-4, w, w, w)
    got, msg = ctx.selftest_resident_wait(code)
    assert got == 4 and str(code - 10) in msg, (got, msg)
    ctx.synchronize()  # (reported once)
    after = ctx.leapfrog(0, 3, 1e-4, w, w, w)
    assert all(np.array_equal(before[k], after[k]) for k in ("w_next", "mom_next", "grad_cur", "loglik"))
    ctx.close()
    small = m.Context(m.baseline_config(precision=m.PREC_FP32), 1, 1024)
    small.set_window_data(0, x[:1024], y[:1024])
    assert small.selftest_resident_wait(code)[0] == 1   # (CTAs of one tile have the evaluations' arithmetic)
    small.close()


@pytest.mark.parametrize("rows", [2000, 4096, 16500, 58368])
def test_rows_that_leave_the_integers_in_every_trajectory(built, monkeypatch, rows):
    """FP32 on the chip, targets with outliers, in the CTAs' first rows too: their rows become floats within a trajectory and integers again at the next
    one's start, in launches of several.  Against one launch per step, as in the test of all launches."""
    m, _ = built
    x, y, _ = m.synth_window(8, 0, rows)
    rng = np.random.default_rng(rows)
    y = y.copy()
    y[rng.random(rows) < 2e-3] += 500
    y[3] -= 2000

    def run():
        ctx = m.Context(m.baseline_config(precision=m.PREC_FP32, leapfrog_steps=3, burn_in=0, adapt_steps=0, sample_capacity=6, trace_iters=6,
                                          eps0=1e-5), 1, rows)
        ctx.set_window_data(0, x, y)
        ctx.run_chain(1)
        ctx.run_chain(5)
        out = ctx.get_samples(0), ctx.get_trace(0), ctx.get_state(0)
        ctx.close()
        return out

    s1, t1, g1 = run()
    monkeypatch.setenv("MCMC_B200_NO_MULTISTEP", "1")
    s2, t2, g2 = run()
    assert t1["accepted"].any() and np.array_equal(t1["accepted"], t2["accepted"])
    assert np.abs(s1 - s2).max() <= 1e-5 * np.abs(s2).max()
    assert np.abs(g1["grad"] - g2["grad"]).max() <= 1e-5 * np.abs(g2["grad"]).max()


@pytest.mark.parametrize("rows", [16500, 58368])
@pytest.mark.parametrize("eps0", [1e19, 1e30])
def test_a_diverging_trajectory_by_integers_rejects_and_the_chain_stays(built, eps0, rows):
    """As test_a_diverging_trajectory_rejects_and_the_chain_stays, with more than a tile in a CTA."""
    m, _ = built
    x, y, _ = m.synth_window(8, 0, rows)
    ctx = m.Context(m.baseline_config(precision=m.PREC_FP32, leapfrog_steps=8, sample_capacity=4, trace_iters=4, eps0=eps0), 1, rows)
    ctx.set_window_data(0, x, y)
    ctx.run_chain(4)
    assert not ctx.get_trace(0)["accepted"].any() and not ctx.get_samples(0).any()   # the chain's start, w = 0
    assert np.abs(ctx.leapfrog(0, 1, 0.0, *[np.zeros(P, np.float32)] * 3)["grad_cur"] - ctx.get_state(0)["grad"]).max() <= 1e-5 * np.abs(ctx.get_state(0)["grad"]).max()
    ctx.close()


@pytest.mark.parametrize("rows", [1025, 4096, 16500, 61440])
def test_steps_of_one_call_are_those_of_several_calls_but_for_rounding(built, rows):
    """FP32: a step's range comes from the step before it or, first in a call, from its own rows, or it goes by FFMA; whole calls have the same bits again.
    Gradients by either are off by 2^-21 of their terms' root sum of squares at most (test_gpu_split.py), which is below the largest of a gradient's values here:
    1e-6 of it for two of them."""
    m, _ = built
    x, y, _ = m.synth_window(7, 0, rows)
    ctx = m.Context(m.reference_config(precision=0, sample_capacity=0), 1, rows)
    ctx.set_window_data(0, x, y)
    rng = np.random.default_rng(rows)
    w, mom = (0.15 * rng.standard_normal(P)).astype(np.float32), rng.standard_normal(P).astype(np.float32)
    start = ctx.potential_and_grad(0, w)["grad"]
    whole, again = (ctx.leapfrog(0, 6, 1e-5, w, mom, start) for _ in range(2))
    assert np.array_equal(whole["grad_cur"], again["grad_cur"]) and np.array_equal(whole["w_next"], again["w_next"])
    for L in (1, 2, 3):
        s = {"w_next": w, "mom_next": mom, "grad_cur": start}
        for _ in range(6 // L):
            s = ctx.leapfrog(0, L, 1e-5, s["w_next"], s["mom_next"], s["grad_cur"])
        assert np.abs(s["grad_cur"] - whole["grad_cur"]).max() <= 1e-6 * np.abs(whole["grad_cur"]).max()
    ctx.close()


@pytest.mark.parametrize("rows", [1000, 1025, 4096, 16500, 58368])
def test_a_calls_only_step_ends_with_the_evaluations_gradient(built, rows):
    """FP32, calls of one step: the tile arithmetic of evaluations, whose bits hang on nothing but the position; captured in a graph before anything
    else has run it, with row losses, in place."""
    import torch
    m, _ = built
    ctx = m.Context(m.reference_config(precision=0, sample_capacity=0), 1, rows)
    x, y, _ = m.synth_window(8, 0, rows)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    p, out, keep = _step_args(m, torch, ctx, xd, yd, False)
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.mcmc_step(*p, 1, 1e-3, stream=s.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    got = [v.cpu().numpy() for v in out]
    ctx.set_window_data(0, x, y)
    at = ctx.potential_and_grad(0, got[0], want_row_loss=True)
    assert np.array_equal(got[2], at["grad"]) and np.array_equal(got[4][:rows], at["row_loss"])
    del graph
    p, out, keep = _step_args(m, torch, ctx, xd, yd, True)
    ctx.mcmc_step(*p, 1, 1e-3)
    ctx.synchronize()
    for a, b in zip(got, out):
        assert np.array_equal(a, b.cpu().numpy())
    h = [v.cpu().numpy() for v in _step_args(m, torch, ctx, xd, yd, False)[2][:3]]
    one = ctx.leapfrog(0, 1, 1e-3, *h)
    assert np.array_equal(one["w_next"], got[0]) and np.array_equal(one["grad_cur"], got[2])
    ctx.close()
