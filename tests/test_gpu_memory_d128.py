"""GPU: the memory rules at head dimension 128 vs the CPU oracle. A problem's rows are divided over 8 CTAs
where all CTAs of the launch then find room at once, else over 4: the problem counts lie on both sides of that
line for every rule, the lengths on both sides of a backward (8) and a forward (16) tile. Tolerances as in the
tests of the other head dimensions; a second pass must give the same bits (the sums over CTAs have one order)."""
import numpy as np
import pytest

from helpers import make_problem, oracle_chunkwise, oracle_exact, rel_err, to_dev

pytestmark = pytest.mark.gpu

REL = 1e-4
DIM = 128
RULES = {0: "delta", 1: "titans", 2: "hebbian"}


@pytest.fixture(scope="module")
def D():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from nl_hecate_b200 import dispatch
    return dispatch


def _np(t):
    return t.detach().cpu().numpy()


def _keys(rule):
    return (["d_k", "d_v", "d_q", "d_alpha", "d_m_initial"] + (["d_theta"] if rule != 2 else []) +
            (["d_eta", "d_s_initial"] if rule == 1 else []))


def _twice(f):
    """f() run twice into fresh buffers; the bits of every output agree."""
    a, b = f(), f()
    for key in a:
        if a[key] is not None:
            assert np.array_equal(_np(a[key]), _np(b[key])), key
    return a


# chunk 0: the exact rule on checkpoints every `interval` tokens, recomputed window by window
@pytest.mark.parametrize("rule,n,s,interval,chunk", [
    (0, 1, 33, 1000, 0), (0, 3, 17, 5, 0), (0, 20, 9, 9, 0), (0, 37, 7, 3, 0), (0, 38, 17, 8, 0), (0, 40, 9, 1, 0),
    (1, 1, 33, 1000, 0), (1, 3, 17, 5, 0), (1, 16, 9, 9, 0), (1, 19, 9, 4, 0), (1, 37, 7, 3, 0), (1, 40, 17, 8, 0),
    (2, 1, 33, 1000, 0), (2, 3, 17, 5, 0), (2, 40, 9, 4, 0),
    (0, 2, 33, 3, 3), (0, 2, 70, 64, 64), (0, 40, 33, 16, 16),
    (1, 2, 33, 3, 3), (1, 2, 70, 64, 64), (1, 19, 33, 16, 16), (1, 40, 33, 16, 16)])
def test_recompute_pair(D, orc, rule, n, s, interval, chunk):
    p = make_problem(orc, n, s, DIM, 6100 + n + s + interval, "rand")
    w = oracle_chunkwise(orc, RULES[rule], p, chunk) if chunk else oracle_exact(orc, RULES[rule], p)
    t = to_dev(p)
    mc, sc, y = D.rule_forward(rule, t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], t["m0"], t["s0"],
                               interval, chunk)
    assert rel_err(_np(y), w["y"]) <= REL
    g = _twice(lambda: D.rule_backward(rule, t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], mc, sc,
                                       t["dy"], interval, chunk))
    for key in _keys(rule):
        assert rel_err(_np(g[key]), w[key]) <= REL, key


@pytest.mark.parametrize("rule,n,s", [(0, 1, 1), (0, 2, 33), (0, 37, 7), (0, 38, 17), (1, 1, 1), (1, 2, 33), (1, 16, 9),
                                      (1, 19, 17), (1, 37, 9), (1, 40, 8)])
def test_exact_pair(D, orc, rule, n, s):
    """Stored trajectories; d_m_initial and d_s_initial are added up over the problems in arrival order."""
    p = make_problem(orc, n, s, DIM, 6300 + n + s, "rand")
    w = oracle_exact(orc, RULES[rule], p)
    t = to_dev(p)
    if rule == 1:
        ms, ss, y = D.titans_forward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], t["m0"], t["s0"])
        f = lambda: D.titans_backward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], ms, ss, t["dy"])
        assert rel_err(_np(ss), w["s_states"]) <= REL
    else:
        ms, y = D.delta_forward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["m0"])
        f = lambda: D.delta_backward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], ms, t["dy"])
    assert rel_err(_np(y), w["y"]) <= REL and rel_err(_np(ms), w["m_states"]) <= REL
    initial = ("d_m_initial", "d_s_initial")
    g = f()
    _twice(lambda: {k: v for k, v in f().items() if k not in initial})
    for key in _keys(rule):
        assert rel_err(_np(g[key]), w[key].sum(0) if key in initial else w[key]) <= REL, key


@pytest.mark.parametrize("rule", [0, 1, 2])
@pytest.mark.parametrize("t0,t1", [(0, 19), (5, 14), (8, 16), (18, 19), (7, 7)])
def test_segment_backward_leaves_the_other_tokens_alone(D, orc, rule, t0, t1):
    """A segment's gradients with seeds of zero are those of a sequence of its own; nothing outside it is written.
    An empty segment hands its seed on."""
    import torch
    s, L = 19, t1 - t0
    t = to_dev(make_problem(orc, 1, s, DIM, 6500 + t0, "rand"))
    sl = {k: (v[:, t0:t1].contiguous() if k not in ("m0", "s0") else v) for k, v in t.items()}
    seed = torch.zeros(1, DIM * DIM, device="cuda") if L else torch.full((1, DIM * DIM), 2.0, device="cuda")
    out = {k: torch.full_like(t["k"], 7.0) for k in ("d_k_mem", "d_v_mem", "d_q_mem")}
    out.update({k: torch.full_like(t["alpha"], 7.0) for k in ("d_alpha", "d_theta", "d_eta")})
    out.update(d_m_out=torch.empty(1, DIM * DIM, device="cuda"), d_s_out=torch.empty(1, DIM * DIM, device="cuda"))
    ref = None
    ms = ss = torch.zeros(1, DIM * DIM, device="cuda")
    if L:
        ms, ss, _ = D.rule_forward(rule, *(sl[k] for k in ("k", "v", "q", "alpha", "theta", "eta", "m0", "s0")), 1)
        name = {0: "delta", 1: "titans", 2: "hebbian"}[rule]
        q = {k: _np(v) for k, v in sl.items()}
        ref = oracle_exact(orc, name, q)
    args = dict(k_mem=t["k"], v_mem=t["v"], q_mem=t["q"], alpha=t["alpha"], m_states=ms, d_y=t["dy"], d_m_seed=seed,
                t_start=t0, t_end=t1, d=DIM, batch_size=1, seq_len=s)
    use = ["d_k_mem", "d_v_mem", "d_q_mem", "d_alpha", "d_m_out"]
    entry = "hebbian_backward_segment_f32_cuda"
    if rule != 2:
        entry = "delta_backward_segment_f32_cuda"
        args.update(theta=t["theta"], error_clip=0.0)
        use.append("d_theta")
    if rule == 1:
        entry = "titans_backward_segment_f32_cuda"
        args.update(eta=t["eta"], s_states=ss, d_s_seed=seed)
        use += ["d_eta", "d_s_out"]
    D.call(entry, **args, **{k: out[k] for k in use})
    for key in use:
        got = _np(out[key])
        if key in ("d_m_out", "d_s_out"):
            if L:
                want = ref["d_m_initial" if key == "d_m_out" else "d_s_initial"]
                assert rel_err(got, want) <= REL, key
            else:
                assert (got == 2.0).all(), key
            continue
        assert (got[:, :t0] == 7.0).all() and (got[:, t1:] == 7.0).all(), key
        if L:
            assert rel_err(got[:, t0:t1], ref[key.replace("_mem", "")]) <= REL, key


@pytest.mark.parametrize("n,s", [(2, 5), (3, 37), (19, 16), (40, 33)])
def test_both_stagings_of_the_forward_give_the_same_bits(D, orc, n, s):
    """NLH_OPT_BULK_STAGING = 0: cp.async in place of bulk copies, exact and frozen, both splits."""
    t = to_dev(make_problem(orc, n, s, DIM, 6600 + n + s, "rand"))
    out = []
    for on in (1, 0):
        D.call("nlh_set_option", option=5, value=on)
        try:
            out.append([x for rule, chunk in ((0, 0), (1, 0), (2, 0), (0, 8), (1, 8)) for x in
                        D.rule_forward(rule, *(t[k] for k in ("k", "v", "q", "alpha", "theta", "eta", "m0", "s0")), 8, chunk)
                        if x is not None])
        finally:
            D.call("nlh_set_option", option=5, value=1)
    for x, y in zip(*out):
        assert np.array_equal(_np(x), _np(y))
    assert D.call("nlh_bulk_timeout_flag") == 0


def test_clipped_rule_at_the_same_size_runs_the_generic_kernels(D, orc):
    p = make_problem(orc, 2, 12, DIM, 6700, "const", scale=1.0, state_scale=1.0)
    w = oracle_exact(orc, "titans", p, error_clip=1.0, m_norm_max=5.0)
    t = to_dev(p)
    ms, ss, y = D.titans_forward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], t["m0"], t["s0"],
                                    error_clip=1.0, m_norm_max=5.0)
    assert rel_err(_np(y), w["y"]) <= REL and rel_err(_np(ms), w["m_states"]) <= REL
    g = D.titans_backward_dd(t["k"], t["v"], t["q"], t["alpha"], t["theta"], t["eta"], ms, ss, t["dy"], error_clip=1.0)
    for key in ["d_k", "d_v", "d_q", "d_alpha", "d_theta", "d_eta"]:
        assert rel_err(_np(g[key]), w[key]) <= REL, key
