"""The work a user has this library do, as cases that can be timed: one evaluation of the log density and its
gradient, the drop-in leapfrog trajectory with its accept ratio, whole chains from one window to two hundred in
both precisions and both hidden widths, prediction from stored samples, and one window taken from host data to
its posterior.  Everything goes through the public entry points of ``mcmc_bnn_example_b200``.

A case is a plain dict; ``kind`` says which of the five flows below it is:

grad     ``potential_and_grad``: host parameters in, log density, gradient and (optionally) row losses out
step     ``mcmc_step`` + ``log_acpt`` on device pointers, the inner loop of a program written against the
         reference's header interface
chain    ``reset_chain``, ``run_chain`` of ``iters`` HMC iterations on every window, the samples of every window
         and the last window's state read back
predict  ``predict_mean`` of ``count`` stored samples on ``rows`` host rows
pass     one of a sequence of windows: ``set_window_data`` from host arrays, a fresh chain, its samples and
         ``final_loss``
"""
import math

import numpy as np
import torch

import mcmc_bnn_example_b200 as m

D = 22
WINDOW_ROWS = 58368           # the reference's window
ON_CHIP = 126e6               # bytes of L2: a dataset below this need not come from memory for every gradient
MAX_ROW_GRADS = 2.3e9         # rows x gradients of the largest listed chain (200 windows x 58368 rows x 200)


def _eps(case):
    """Step sizes at which trajectories of the two likelihoods keep their energy (the Gaussian one's forces grow with
    the rows): nearly every proposal is accepted, so that a chain's path does not hang on the last bits of an accept
    ratio."""
    return 1e-3 if case["likelihood"] == "student_t" else min(5e-5, 3.0 / case["rows"])


def listed():
    return [
        # a log-density probe on a small dataset: nothing but latency (unit tests, tuning scripts, tiny models)
        {"name": "grad_1000_fp32", "kind": "grad", "rows": 1000, "hidden": 40, "precision": "fp32",
         "likelihood": "gaussian", "row_loss": False},
        # the same call on the reference's window, with the row losses a diagnostic plot wants
        {"name": "grad_window_tf32", "kind": "grad", "rows": WINDOW_ROWS, "hidden": 40, "precision": "tf32",
         "likelihood": "student_t", "row_loss": True},
        # the reference's own inner loop (mcmc_step<float, 10> and log_acpt_prec) on its window, FP32 build
        {"name": "step_window_fp32", "kind": "step", "rows": WINDOW_ROWS, "hidden": 40, "precision": "fp32",
         "likelihood": "student_t", "steps": 10},
        # ... and its TF32 build on a shorter window whose last tile is ragged
        {"name": "step_ragged_tf32", "kind": "step", "rows": 30011, "hidden": 40, "precision": "tf32",
         "likelihood": "gaussian", "steps": 10},
        # the reference's preset: one window, FP32, 1000 leapfrog steps to an iteration
        {"name": "chain_reference_fp32", "kind": "chain", "windows": 1, "rows": WINDOW_ROWS, "hidden": 40,
         "precision": "fp32", "likelihood": "student_t", "steps": 1000, "iters": 2},
        # one window's chain with short trajectories, TF32: a string of short dependent launches
        {"name": "chain_one_tf32", "kind": "chain", "windows": 1, "rows": WINDOW_ROWS, "hidden": 40,
         "precision": "tf32", "likelihood": "gaussian", "steps": 10, "iters": 100},
        # one GPU's share of 200 windows on an eight-GPU box
        {"name": "chain_25_tf32", "kind": "chain", "windows": 25, "rows": WINDOW_ROWS, "hidden": 40,
         "precision": "tf32", "likelihood": "gaussian", "steps": 10, "iters": 40},
        # the benchmark's workload: 200 windows on one GPU
        {"name": "chain_200_tf32", "kind": "chain", "windows": 200, "rows": WINDOW_ROWS, "hidden": 40,
         "precision": "tf32", "likelihood": "gaussian", "steps": 10, "iters": 20},
        # a batch of ragged windows in FP32
        {"name": "chain_16_fp32", "kind": "chain", "windows": 16, "rows": 40013, "hidden": 40,
         "precision": "fp32", "likelihood": "student_t", "steps": 10, "iters": 20},
        # one GPU's share of the wide model's stress test on an eight-GPU box
        {"name": "chain_wide_tf32", "kind": "chain", "windows": 8, "rows": 1048576, "hidden": 128,
         "precision": "tf32", "likelihood": "gaussian", "steps": 10, "iters": 2},
        # posterior-mean prediction of a full set of samples on a window's rows
        {"name": "predict_800", "kind": "predict", "rows": WINDOW_ROWS, "hidden": 40, "precision": "tf32",
         "likelihood": "student_t", "count": 800},
        # a new window arrives on the host and leaves as samples and a mean loss
        {"name": "pass_window_tf32", "kind": "pass", "rows": WINDOW_ROWS, "hidden": 40, "precision": "tf32",
         "likelihood": "student_t", "steps": 10, "iters": 60},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grad", "step", "chain", "chain", "chain", "predict", "pass"])
    case = {"kind": kind, "hidden": 40 if rng.random() < 0.75 else 128, "precision": rng.choice(["fp32", "tf32"]),
            "likelihood": rng.choice(["gaussian", "student_t"])}
    wide = 3.3 if case["hidden"] == 128 else 1.0
    slow = wide * (4.5 if case["precision"] == "fp32" else 1.0)
    if kind == "grad":
        case.update(rows=_log(rng, 100, 300000), row_loss=rng.random() < 0.5)
    elif kind == "step":
        case.update(rows=_log(rng, 1000, 200000), steps=_log(rng, 1, 40))
    elif kind == "chain":
        rows = _log(rng, 2000, 1048576)
        windows = min(_log(rng, 1, 200), max(1, 12000000 // rows))
        grads = min(2000.0, max(10.0, MAX_ROW_GRADS * rng.uniform(0.05, 0.9) / slow / (rows * windows)))
        # (long trajectories belong to the reference's preset; under the Gaussian one they amplify rounding)
        steps = max(2, min(_log(rng, 5, 1000 if case["likelihood"] == "student_t" else 40), int(grads)))
        iters = max(1, min(60, int(grads / steps)))
        case.update(rows=rows, windows=windows, steps=steps, iters=iters)
    elif kind == "predict":
        case.update(rows=_log(rng, 500, WINDOW_ROWS), count=_log(rng, 20, 800 if wide == 1.0 else 200))
    else:
        case.update(rows=_log(rng, 4000, 100000), steps=_log(rng, 5, 20), iters=_log(rng, 10, 60))
    return case


def _config(case, seed, **kw):
    student = case["likelihood"] == "student_t"
    make = m.reference_config if student else m.baseline_config
    return make(H=case["hidden"], precision=m.PREC_TF32 if case["precision"] == "tf32" else m.PREC_FP32,
                eps0=_eps(case), burn_in=0, adapt_steps=0, seed=seed, **kw)


def _window(gen, rows, hidden):
    """X ~ N(0,1), targets of a teacher network with N(0, 0.3^2) weights plus N(0, 0.05^2) noise."""
    dev = "cuda"
    x = torch.randn(rows, D, device=dev, generator=gen)
    w0 = 0.3 * torch.randn(D, hidden, device=dev, generator=gen)
    b0 = 0.3 * torch.randn(hidden, device=dev, generator=gen)
    w1 = 0.3 * torch.randn(hidden, device=dev, generator=gen)
    y = torch.tanh(x @ w0 + b0) @ w1 + 0.3 * torch.randn(1, device=dev, generator=gen)
    return x, y + 0.05 * torch.randn(rows, device=dev, generator=gen)


def _fill(ctx, gen, case):
    for w in range(ctx.n_windows):
        x, y = _window(gen, ctx.rows, case["hidden"])
        torch.cuda.synchronize()
        ctx.set_window_data_ptr(w, x.data_ptr(), y.data_ptr(), True)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, rows = case["kind"], case["rows"]
    if kind == "grad":
        ctx = m.Context(_config(case, seed, sample_capacity=0), 1, rows)
        _fill(ctx, gen, case)
        w = 0.2 * torch.randn(ctx.P, device="cuda", generator=gen)
        return {"case": case, "ctx": ctx, "w": w.cpu().numpy()}
    if kind == "step":
        ctx = m.Context(_config(case, seed, sample_capacity=0), 1, rows)
        x, y = _window(gen, rows, case["hidden"])
        P = ctx.P
        b = {k: torch.zeros(P, device="cuda") for k in
             ("w_prev", "w_next", "mom_prev", "mom_next", "grad_prev", "grad_cur", "grad_next")}
        b["w_prev"] += 0.2 * torch.randn(P, device="cuda", generator=gen)
        b["mom_prev"] += torch.randn(P, device="cuda", generator=gen)
        loss_prev, loss_new = (torch.zeros(rows + P, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        # losses and gradient at the starting point: one step of size zero
        zero = torch.zeros(P, device="cuda")
        torch.cuda.synchronize()
        ctx.mcmc_step(x.data_ptr(), y.data_ptr(), b["w_prev"].data_ptr(), b["w_next"].data_ptr(), zero.data_ptr(),
                      b["mom_next"].data_ptr(), zero.data_ptr(), b["grad_prev"].data_ptr(), b["grad_next"].data_ptr(),
                      loss_prev.data_ptr(), 1, 0.0)
        torch.cuda.synchronize()
        return {"case": case, "ctx": ctx, "x": x, "y": y, "b": b, "loss_prev": loss_prev, "loss_new": loss_new}
    if kind == "chain":
        ctx = m.Context(_config(case, seed, leapfrog_steps=case["steps"], sample_capacity=case["iters"]),
                        case["windows"], rows)
        _fill(ctx, gen, case)
        return {"case": case, "ctx": ctx}
    if kind == "predict":
        # a stored posterior: `count` samples of a short chain on a small window of the same model
        ctx = m.Context(_config(case, seed, leapfrog_steps=40, sample_capacity=case["count"]), 1, 128)
        _fill(ctx, gen, case)
        ctx.run_chain(case["count"])
        xs = torch.randn(rows, D, device="cuda", generator=gen)
        return {"case": case, "ctx": ctx, "xs": xs.cpu().numpy()}
    ctx = m.Context(_config(case, seed, leapfrog_steps=case["steps"], sample_capacity=case["iters"]), 1, rows)
    x, y = _window(gen, rows, case["hidden"])
    return {"case": case, "ctx": ctx, "x": x.cpu().numpy(), "y": y.cpu().numpy()}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "grad":
        return ctx.potential_and_grad(0, state["w"], want_row_loss=case["row_loss"])
    if kind == "step":
        b, eps = state["b"], _eps(case)
        ctx.mcmc_step(state["x"].data_ptr(), state["y"].data_ptr(), b["w_prev"].data_ptr(), b["w_next"].data_ptr(),
                      b["mom_prev"].data_ptr(), b["mom_next"].data_ptr(), b["grad_prev"].data_ptr(),
                      b["grad_cur"].data_ptr(), b["grad_next"].data_ptr(), state["loss_new"].data_ptr(),
                      case["steps"], eps)
        log_acpt = ctx.log_acpt(state["loss_prev"].data_ptr(), state["loss_new"].data_ptr(),
                                state["loss_new"].numel(), b["mom_prev"].data_ptr(), b["mom_next"].data_ptr(),
                                b["grad_cur"].data_ptr(), eps)
        # (the ratio beside the expected kinetic energy: an energy difference is known no better than the energies)
        return {"w": b["w_next"], "mom": b["mom_next"], "grad": b["grad_cur"], "grad_next": b["grad_next"],
                "loss": state["loss_new"], "log_acpt": np.array([log_acpt, 0.5 * ctx.P])}
    if kind == "predict":
        return ctx.predict_mean(0, state["xs"])
    if kind == "pass":
        ctx.set_window_data(0, state["x"], state["y"])
    ctx.reset_chain()
    ctx.run_chain(case["iters"])
    if kind == "pass":
        loglik, logprior = ctx.final_loss(0)
        return {"samples": ctx.get_samples(0), "loglik": loglik, "logprior": logprior}
    samples = np.empty((ctx.n_windows, case["iters"], ctx.P), np.float32)
    for w in range(ctx.n_windows):
        ctx.get_samples(w, out=samples[w])
    return {"samples": samples, "state": ctx.get_state(ctx.n_windows - 1)}


def work(case):
    """Inputs read once and outputs written once; a dataset too large for the chip once for every gradient."""
    H, rows = case["hidden"], case["rows"]
    P = m.num_params(D, H)
    fwd, bwd = 2 * (D + 1) * H + 3 * H, 2 * (D + 1) * H + 7 * H      # per row, a tanh as one operation
    data = 4.0 * rows * (D + 1)
    if case["kind"] == "grad":
        return {"bytes": data + 4.0 * (2 * P + (rows if case["row_loss"] else 0)), "flops": float(rows * (fwd + bwd))}
    if case["kind"] == "predict":
        return {"bytes": 4.0 * rows * (D + 1) + 4.0 * case["count"] * P, "flops": float(rows * case["count"] * fwd)}
    windows, iters = case.get("windows", 1), case.get("iters", 1)
    grads = case["steps"] * iters
    out = 4.0 * (rows + 6 * P) if case["kind"] == "step" else 4.0 * windows * iters * P
    reads = 1 if data * windows < ON_CHIP else grads
    more = rows * iters * fwd if case["kind"] == "pass" else 0       # final_loss
    return {"bytes": data * windows * reads + out, "flops": float(windows * rows * grads * (fwd + bwd) + more)}


def tolerance(case):
    if case["kind"] == "predict":        # FP32 whatever the chain ran in
        return {"rel": 2e-5}
    return {"rel": 2e-3} if case["precision"] == "tf32" else {"rel": 2e-5}
