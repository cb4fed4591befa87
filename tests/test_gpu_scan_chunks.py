"""Recurrences of a prompt step by chunks of tokens on the tensor cores, alone, against a loop over the tokens in 64-bit
and beside the kernels that visit the tokens one by one: at the chunks' edges, over several sequences of unequal length, with
decays from none to all, and with numbers that are not finite."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _batch(lens):
    from prelude_b200.engine.batch import StepItem, build_step_batch
    return build_step_batch([StepItem(i, [0] * n, 0) for i, n in enumerate(lens)], {}, list(range(len(lens)))[::-1],
                            torch.device(DEV), 2, 1 << 20)


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


def _ssm_inputs(lens, H, P, N, groups, seed, step):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    T = sum(lens)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=DEV)

    u = normal(T, H * P + 2 * groups * N).bfloat16()
    dt = normal(T, H + 3).bfloat16()[:, :H]
    bias = torch.full((H,), math.log(math.expm1(step)), device=DEV) + 0.3 * normal(H)
    a_log = torch.log(torch.rand(H, generator=gen, device=DEV) * 15 + 1)
    return u, dt, bias, a_log, normal(H), normal(len(lens), H, N, P)


def _ssm_exact(u, dt, bias, a_log, skip, state, lens, groups):
    R, H, N, P = state.shape
    u, S, inner, at = u.double(), state.double().clone(), H * P, 0
    step = torch.nn.functional.softplus(dt.double() + bias.double(), threshold=50)
    decay = torch.exp(-torch.exp(a_log.double()) * step)
    y = torch.empty(u.shape[0], H, P, dtype=torch.float64, device=DEV)
    for r, n in enumerate(lens):
        slot = R - 1 - r
        for t in range(at, at + n):
            x = u[t, :inner].view(H, P)
            B, C = (u[t, inner + k * groups * N:inner + (k + 1) * groups * N].view(groups, N).repeat_interleave(H // groups, 0) for k in (0, 1))
            S[slot] = decay[t].view(H, 1, 1) * S[slot] + (step[t].view(H, 1) * B).unsqueeze(2) * x.unsqueeze(1)
            y[t] = (S[slot] * C.unsqueeze(2)).sum(1) + skip.double().view(H, 1) * x
        at += n
    return y.view(-1, inner), S


@pytest.fixture(autouse=True)
def _chunks_whatever_the_length(monkeypatch):
    from prelude_b200.ops import kernels as K
    for name in ("SCAN_CHUNKED_MIN_TOKENS", "DELTA_CHUNKED_MIN_TOKENS", "GLA_CHUNKED_MIN_TOKENS"):
        monkeypatch.setattr(K, name, 1)


def _by_tokens(monkeypatch, K):
    """The same call through the kernel that visits the tokens one by one."""
    for name in ("SCAN_CHUNKED_MIN_TOKENS", "DELTA_CHUNKED_MIN_TOKENS", "GLA_CHUNKED_MIN_TOKENS"):
        monkeypatch.setattr(K, name, 1 << 30)


@pytest.mark.parametrize("lens,H,P,N,groups", [
    ([64], 8, 64, 128, 8), ([65, 1, 63], 4, 32, 128, 2), ([127, 40], 2, 16, 64, 1), ([33], 4, 64, 64, 4),
    ([300, 17, 128], 64, 64, 128, 8), ([500], 128, 64, 128, 8), ([200], 3, 48, 128, 3), ([1000], 8, 128, 128, 1)])
@pytest.mark.parametrize("step", [1e-3, 0.05, 1.0])
def test_state_space_by_chunks(lens, H, P, N, groups, step, monkeypatch):
    """No farther from 64-bit than token by token, or than the eight roundings of 6e-8 that the longest chain of products in a
    chunk leaves (token by token the state is rounded once a token, so its error grows with the tokens that a decay leaves:
    5e-6 over a thousand tokens that hardly decay)."""
    from prelude_b200.ops import kernels as K
    u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, P, N, groups, 1, step)
    want_y, want_s = _ssm_exact(u, dt, bias, a_log, skip, state, lens, groups)
    chunked, plain = state.clone(), state.clone()
    y = K.ssm_scan(u, dt, bias, a_log, skip, chunked, _batch(lens), groups)
    _by_tokens(monkeypatch, K)
    y0 = K.ssm_scan(u, dt, bias, a_log, skip, plain, _batch(lens), groups)
    errs = [_rel(y, want_y), _rel(chunked, want_s), _rel(y0, want_y), _rel(plain, want_s)]
    print("chunks y %.2e state %.2e, tokens y %.2e state %.2e" % tuple(errs))
    assert errs[0] <= max(errs[2], 8 * 6e-8) and errs[1] <= max(errs[3], 8 * 6e-8)
    assert not torch.equal(y, y0)             # two kernels, not one twice


def test_state_space_by_chunks_with_numbers_that_are_not_finite():
    """An infinity in x spoils its own column from its token on; what lies before it, and other columns, stay as they are."""
    from prelude_b200.ops import kernels as K
    lens, H, P, N, groups = [150], 2, 32, 128, 1
    u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, P, N, groups, 5, 0.05)
    clean = K.ssm_scan(u, dt, bias, a_log, skip, state.clone(), _batch(lens), groups)
    u[70, 3], u[100, P + 5] = float("inf"), float("nan")
    y = K.ssm_scan(u, dt, bias, a_log, skip, state, _batch(lens), groups)
    keep = torch.ones_like(y, dtype=torch.bool)
    keep[70:, 3] = keep[100:, P + 5] = False
    assert torch.equal(y[keep], clean[keep]) and not torch.isfinite(y[~keep]).any()
    assert not torch.isfinite(state[0, 0, :, 3]).any() and torch.isfinite(state[0, 0, :, :3]).all()


def test_state_space_by_chunks_with_decays_that_leave_nothing():
    """Rates so large that a step forgets everything: the output is that of the current token alone."""
    from prelude_b200.ops import kernels as K
    lens, H, P, N, groups = [100], 2, 32, 64, 1
    u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, P, N, groups, 6, 1.0)
    a_log.fill_(30.0)
    want_y, want_s = _ssm_exact(u, dt, bias, a_log, skip, state, lens, groups)
    y = K.ssm_scan(u, dt, bias, a_log, skip, state, _batch(lens), groups)
    assert _rel(y, want_y) < 1e-6 and _rel(state, want_s) < 1e-6


def _delta_inputs(lens, H, G, D, E, seed, step, key_noise=1.0):
    """``key_noise`` below 1: keys that nearly repeat, so that what a token writes takes most of what the one before it wrote."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    T = sum(lens)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=DEV)

    k = key_noise * normal(T, G * D) + (1 - key_noise) * normal(1, G * D)
    u = torch.cat([normal(T, G * D), k, normal(T, H * E)], 1).bfloat16()
    proj = normal(T, 2 * H + 8).bfloat16()
    bias = torch.full((H,), math.log(math.expm1(step)), device=DEV) + 0.3 * normal(H)
    a_log = torch.log(torch.rand(H, generator=gen, device=DEV) * 15 + 1)
    return u, proj[:, :H], proj[:, H:2 * H], a_log, bias, normal(len(lens), H, D, E)


def _delta_exact(u, b, a, a_log, bias, state, lens, G):
    R, H, D, E = state.shape
    u, S, at, T = u.double(), state.double().clone(), 0, u.shape[0]
    q, k, v = u[:, :G * D].view(T, G, D), u[:, G * D:2 * G * D].view(T, G, D), u[:, 2 * G * D:].view(T, H, E)
    q, k = ((x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for x in (q, k))
    beta = torch.sigmoid(b.double())
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a.double() + bias.double(), threshold=50))
    o = torch.empty(T, H, E, dtype=torch.float64, device=DEV)
    for r, n in enumerate(lens):
        slot = R - 1 - r
        for t in range(at, at + n):
            s = decay[t].view(H, 1, 1) * S[slot]
            w = beta[t].view(H, 1) * (v[t] - (s * k[t].unsqueeze(2)).sum(1))
            S[slot] = s + k[t].unsqueeze(2) * w.unsqueeze(1)
            o[t] = (S[slot] * q[t].unsqueeze(2)).sum(1) * D ** -0.5
        at += n
    return o.view(T, H * E), S


@pytest.mark.parametrize("lens,H,G,D,E", [
    ([64], 4, 2, 128, 128), ([65, 1, 63], 4, 4, 64, 32), ([127, 40], 2, 1, 128, 16), ([33], 4, 2, 64, 64), ([1] * 40 + [70], 2, 2, 64, 16),
    ([300, 17, 128], 16, 8, 128, 128), ([500], 32, 16, 128, 128), ([200], 3, 3, 128, 48), ([1000], 2, 1, 128, 32)])
@pytest.mark.parametrize("step,key_noise", [(1e-3, 1.0), (0.05, 1.0), (1.0, 1.0), (1e-3, 0.1)])
def test_gated_delta_rule_by_chunks(lens, H, G, D, E, step, key_noise, monkeypatch):
    """No farther from 64-bit than token by token, or than a few roundings of 6e-8: eight products in the longest chain, and three
    such products one behind the other (into the state, through the inverse, out of the state)."""
    from prelude_b200.ops import kernels as K
    u, b, a, a_log, bias, state = _delta_inputs(lens, H, G, D, E, 2, step, key_noise)
    want_o, want_s = _delta_exact(u, b, a, a_log, bias, state, lens, G)
    chunked, plain = state.clone(), state.clone()
    o = K.gated_delta_scan(u, b, a, a_log, bias, chunked, _batch(lens), G)
    _by_tokens(monkeypatch, K)
    o0 = K.gated_delta_scan(u, b, a, a_log, bias, plain, _batch(lens), G)
    errs = [_rel(o, want_o), _rel(chunked, want_s), _rel(o0, want_o), _rel(plain, want_s)]
    print("chunks o %.2e state %.2e, tokens o %.2e state %.2e" % tuple(errs))
    assert errs[0] <= max(errs[2], 3 * 8 * 6e-8) and errs[1] <= max(errs[3], 3 * 8 * 6e-8)
    assert not torch.equal(o, o0)


def test_gated_delta_rule_by_chunks_with_numbers_that_are_not_finite():
    """An infinity in v spoils its own column from its token on, one in a key every column; what lies before stays as it is."""
    from prelude_b200.ops import kernels as K
    lens, H, G, D, E = [150], 2, 2, 64, 32
    u, b, a, a_log, bias, state = _delta_inputs(lens, H, G, D, E, 5, 0.05)
    clean = K.gated_delta_scan(u, b, a, a_log, bias, state.clone(), _batch(lens), G)
    u[70, 2 * G * D + 3], u[100, G * D + D + 7] = float("inf"), float("nan")
    o = K.gated_delta_scan(u, b, a, a_log, bias, state, _batch(lens), G)
    keep = torch.ones_like(o, dtype=torch.bool)
    keep[70:, 3] = keep[100:, E:] = False
    assert torch.equal(o[keep], clean[keep]) and not torch.isfinite(o[~keep]).any()
    assert not torch.isfinite(state[0, 0, :, 3]).any() and torch.isfinite(state[0, 0, :, :3]).all() and not torch.isfinite(state[0, 1]).any()


def _gla_inputs(lens, H, N, P, seed, low, high):
    """Decays between ``low`` and ``high``, spread over their logarithms."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    T = sum(lens)
    proj = torch.randn(T, 2 * H * N + H * P + 8, generator=gen, device=DEV).bfloat16()
    lo, hi = math.log(low), math.log(high)
    decay = torch.exp(torch.rand(T, H * N, generator=gen, device=DEV) * (hi - lo) + lo)
    state = torch.randn(len(lens), H, N, P, generator=gen, device=DEV)
    return proj[:, :H * N], proj[:, H * N:2 * H * N], proj[:, 2 * H * N:2 * H * N + H * P], decay, state


def _gla_exact(q, k, v, decay, scale, state, lens):
    R, H, N, P = state.shape
    T, S, at = q.shape[0], state.double().clone(), 0
    q, k, v, a = q.double().view(T, H, N), k.double().view(T, H, N), v.double().view(T, H, P), decay.double().view(T, H, N)
    o = torch.empty(T, H, P, dtype=torch.float64, device=DEV)
    for r, n in enumerate(lens):
        slot = R - 1 - r
        for t in range(at, at + n):
            S[slot] = a[t].unsqueeze(2) * S[slot] + k[t].unsqueeze(2) * v[t].unsqueeze(1)
            o[t] = (S[slot] * q[t].unsqueeze(2)).sum(1) * scale
        at += n
    return o.view(T, H * P), S


@pytest.mark.parametrize("lens,H,N,P", [
    ([64], 4, 128, 128), ([17, 1, 15], 4, 64, 32), ([127, 40], 2, 128, 16), ([33], 4, 64, 64), ([1] * 40 + [70], 2, 64, 32),
    ([300, 17, 128], 16, 128, 128), ([500], 32, 128, 128), ([200], 3, 128, 48), ([1000], 2, 64, 96), ([160], 64, 128, 128)])
@pytest.mark.parametrize("low,high", [(0.99, 1.0), (0.9, 1.0), (1e-3, 1.0), (1e-38, 1e-3)])
def test_gated_linear_attention_by_sixteens(lens, H, N, P, low, high, monkeypatch):
    """No farther from 64-bit than token by token, or than the sixteen roundings of 6e-8 that a decay's product over sixteen
    tokens collects."""
    from prelude_b200.ops import kernels as K
    q, k, v, decay, state = _gla_inputs(lens, H, N, P, 3, low, high)
    want_o, want_s = _gla_exact(q, k, v, decay, 0.25, state, lens)
    chunked, plain = state.clone(), state.clone()
    o = K.gla_scan(q, k, v, decay, 0.25, chunked, _batch(lens))
    _by_tokens(monkeypatch, K)
    o0 = K.gla_scan(q, k, v, decay, 0.25, plain, _batch(lens))
    errs = [_rel(o, want_o), _rel(chunked, want_s), _rel(o0, want_o), _rel(plain, want_s)]
    print("sixteens o %.2e state %.2e, tokens o %.2e state %.2e" % tuple(errs))
    assert errs[0] <= max(errs[2], 16 * 6e-8) and errs[1] <= max(errs[3], 16 * 6e-8)
    assert not torch.equal(o, o0)


def test_gated_linear_attention_by_sixteens_with_numbers_that_are_not_finite():
    """An infinity in v spoils its own column from its token on; what lies before it, and other columns, stay as they are.  So
    does one in a key, for every column of its head."""
    from prelude_b200.ops import kernels as K
    lens, H, N, P = [50], 2, 64, 32
    q, k, v, decay, state = _gla_inputs(lens, H, N, P, 5, 0.9, 1.0)
    clean = K.gla_scan(q, k, v, decay, 1.0, state.clone(), _batch(lens))
    v[20, 3], k[37, N + 5] = float("inf"), float("nan")
    o = K.gla_scan(q, k, v, decay, 1.0, state, _batch(lens))
    keep = torch.ones_like(o, dtype=torch.bool)
    keep[20:, 3] = keep[37:, P:] = False
    assert torch.equal(o[keep], clean[keep]) and not torch.isfinite(o[~keep]).any()
    assert not torch.isfinite(state[0, 0, :, 3]).any() and torch.isfinite(state[0, 0, :, :3]).all()


@pytest.mark.parametrize("at", [0, 1, 62, 63, 64, 101])
@pytest.mark.parametrize("kind", ["state space", "gated delta rule, decay", "gated delta rule, beta", "gated linear attention"])
def test_a_step_size_or_decay_that_is_no_number_spoils_no_earlier_token(kind, at):
    """The first or the second token of a pair, at a chunk's edges and inside one: every output of the head from that token on is NaN,
    what lies before it and the other head stay as they are to the last bit."""
    from prelude_b200.ops import kernels as K
    lens = [150]
    if kind == "state space":
        P = 32
        u, dt, bias, a_log, skip, state = _ssm_inputs(lens, 2, P, 64, 1, 5, 0.05)
        poisoned, spoil = dt.clone(), (at, 1)
        run = lambda d, s: K.ssm_scan(u, d, bias, a_log, skip, s, _batch(lens), 1)
    elif kind.startswith("gated delta"):
        P = 16
        u, b, a, a_log, bias, state = _delta_inputs(lens, 2, 2, 64, P, 5, 0.05)
        dt = a if kind.endswith("decay") else b
        poisoned, spoil = dt.clone(), (at, 1)
        run = lambda d, s: K.gated_delta_scan(u, *((b, d) if kind.endswith("decay") else (d, a)), a_log, bias, s, _batch(lens), 2)
    else:
        P = 32
        q, k, v, dt, state = _gla_inputs(lens, 2, 64, P, 5, 0.9, 1.0)
        poisoned, spoil = dt.clone(), (at, 64 + 9)
        run = lambda d, s: K.gla_scan(q, k, v, d, 1.0, s, _batch(lens))
    clean_state, state = state.clone(), state.clone()
    clean = run(dt, clean_state)
    poisoned[spoil] = float("nan")
    y = run(poisoned, state)
    keep = torch.ones_like(y, dtype=torch.bool)
    keep[at:, P:] = False
    assert torch.equal(y[keep], clean[keep]) and torch.isnan(y[~keep]).all()
    assert torch.equal(state[0, 0], clean_state[0, 0])
    gone = state[0, 1, 9] if kind == "gated linear attention" else state[0, 1]
    assert torch.isnan(gone).all()


@pytest.mark.parametrize("odd_state,odd_result", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("kind", ["state space", "gated delta rule", "gated linear attention"])
def test_state_and_result_anywhere(kind, odd_state, odd_result):
    """A result or a state that begins four bytes past a boundary is taken as before there were chunks (by tokens, where the
    chunks' wider accesses do not fit)."""
    from prelude_b200.ops import kernels as K
    lens, H = [40, 70], 2
    if kind == "state space":
        u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, 32, 64, 1, 5, 0.05)
        width, run = H * 32, lambda s, o: K.ssm_scan(u, dt, bias, a_log, skip, s, _batch(lens), 1, out=o)
    elif kind == "gated delta rule":
        u, b, a, a_log, bias, state = _delta_inputs(lens, H, 2, 64, 16, 5, 0.05)
        width, run = H * 16, lambda s, o: K.gated_delta_scan(u, b, a, a_log, bias, s, _batch(lens), 2, out=o)
    else:
        q, k, v, decay, state = _gla_inputs(lens, H, 64, 32, 5, 0.9, 1.0)
        width, run = H * 32, lambda s, o: K.gla_scan(q, k, v, decay, 1.0, s, _batch(lens), out=o)

    def at(shape, odd):
        n = math.prod(shape)
        return torch.zeros(n + 1, device=DEV)[odd:n + odd].view(shape)

    want_s = state.clone()
    want = run(want_s, at((sum(lens), width), False))
    got_s = at(tuple(state.shape), odd_state).copy_(state)
    got = run(got_s, at((sum(lens), width), odd_result))
    assert _rel(got, want.double()) < 1e-6 and _rel(got_s, want_s.double()) < 1e-6


def _scan(kind, lens, H, seed=5):
    """(A call (state, batch) -> result, the state it starts from) over sequences of these lengths."""
    from prelude_b200.ops import kernels as K
    if kind == "state space":
        u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, 64, 64, 1, seed, 0.05)
        return lambda s, b: K.ssm_scan(u, dt, bias, a_log, skip, s, b, 1), state
    if kind == "gated delta rule":
        u, b_, a, a_log, bias, state = _delta_inputs(lens, H, H, 64, 128, seed, 0.05)
        return lambda s, b: K.gated_delta_scan(u, b_, a, a_log, bias, s, b, H), state
    q, k, v, decay, state = _gla_inputs(lens, H, 128, 128, seed, 0.9, 1.0)
    return lambda s, b: K.gla_scan(q, k, v, decay, 1.0, s, b), state


KINDS = ["state space", "gated delta rule", "gated linear attention"]


def _thresholds(monkeypatch, tokens, lengths=(1, 0, 1)):
    from prelude_b200.ops import kernels as K
    for name in ("SCAN_CHUNKED_MIN_TOKENS", "DELTA_CHUNKED_MIN_TOKENS", "GLA_CHUNKED_MIN_TOKENS"):
        monkeypatch.setattr(K, name, tokens)
    monkeypatch.setattr(K, "DELTA_CHUNKED_LENGTHS", lengths)


@pytest.mark.parametrize("lens,limit", [([1] * 60 + [30], 70), ([1, 24, 1, 70, 23, 24], 70), ([1, 24, 70, 23, 24], 1), ([23] * 5, 70), ([24, 100], 1),
                                        ([1] * 130 + [90] + [1] * 130, 70)])
def test_every_sequence_of_the_delta_rule_runs_as_its_own_length_asks(lens, limit, monkeypatch):
    """Sequences of one token beside portions: where more than two have fewer than 24, those of 70 run by chunks, the others
    token by token - to the last bit what each gives where all run one way."""
    run, state = _scan("gated delta rule", lens, 2)
    results = []
    for tokens, lengths in ((1 << 30, (1, 0, 1)), (1, (1, 0, 1)), (24, (24, 2, 70))):
        _thresholds(monkeypatch, tokens, lengths)
        s = state.clone()
        results.append((run(s, _batch(lens)), s))
    (y_tok, s_tok), (y_chunk, s_chunk), (y, s) = results
    at = 0
    for r, n in enumerate(lens):
        want_y, want_s = (y_chunk, s_chunk) if n >= limit else (y_tok, s_tok)
        slot = len(lens) - 1 - r
        assert torch.equal(y[at:at + n], want_y[at:at + n]) and torch.equal(s[slot], want_s[slot])
        at += n


@pytest.mark.parametrize("lens", [[1] * 60 + [30], [1, 24, 1, 70, 2, 24, 1], [1] * 130 + [90] + [1] * 130])
def test_single_tokens_of_a_state_space_step_run_as_a_decode_step_does(lens, monkeypatch):
    """Sequences of one token beside portions: to the last bit what a step of single tokens alone gives them."""
    from prelude_b200.ops import kernels as K
    _thresholds(monkeypatch, 24)
    H = 2
    u, dt, bias, a_log, skip, state = _ssm_inputs(lens, H, 64, 64, 1, 5, 0.05)
    alone, at = state.clone(), [sum(lens[:r]) for r, n in enumerate(lens) if n == 1]
    b = _batch([1] * len(at))
    b.state_slots = torch.tensor([len(lens) - 1 - r for r, n in enumerate(lens) if n == 1], dtype=torch.int32, device=DEV)
    want = K.ssm_scan(u[at].contiguous(), dt[at].contiguous(), bias, a_log, skip, alone, b, 1)
    got = K.ssm_scan(u, dt, bias, a_log, skip, state, _batch(lens), 1)
    slots = b.state_slots.long()
    assert torch.equal(got[at], want) and torch.equal(state[slots], alone[slots])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("H", [2, 16, 64])
@pytest.mark.parametrize("lens", [[70], [30, 40], [1] * 20 + [64], [1, 24, 1, 70, 23, 24, 50], [3, 5], [24] * 9, [2] * 60, [1, 1, 70], [1, 1, 1, 70, 80]])
@pytest.mark.parametrize("room", [16, 256])
def test_a_recorded_step_runs_what_a_launched_one_does(kind, H, lens, room, monkeypatch):
    """Room for more requests than there are and lengths that are known on the device alone: the same routes and slices, to the last
    bit; rows behind the last request, whose lengths are not positive, are nobody's."""
    if len(lens) > room:
        pytest.skip("more requests than rows")
    _thresholds(monkeypatch, 24, (24, 2, 60))
    pad = 13
    run, state = _scan(kind, lens + [pad], H)              # the last sequence's tokens are the recorded step's padding
    plain, launched, full = state.clone(), _batch(lens + [pad]), _batch(lens + [pad])
    launched.cu_q, launched.state_slots, launched.q_lens = launched.cu_q[:-1].clone(), launched.state_slots[:-1].clone(), launched.q_lens[:-1]
    y = run(plain, launched)

    def with_room(t, n):
        return torch.cat([t, torch.zeros(n - t.numel(), dtype=t.dtype, device=DEV)])

    full.cu_q, full.state_slots = with_room(launched.cu_q, room + 1), with_room(launched.state_slots, room)
    full.extras["recorder"] = object()
    again = state.clone()
    got = run(again, full)
    assert torch.equal(got[:sum(lens)], y[:sum(lens)]) and torch.equal(again, plain)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("first", [[1] * 20 + [100, 80], [10] * 2 + [9] * 20, [180] + [0] * 20 + [20], [9] * 21 + [11]])
def test_a_captured_call_serves_other_lengths(kind, first, monkeypatch):
    """A graph of the call, replayed after the cumulative lengths have been filled anew: the same as a call of its own."""
    _thresholds(monkeypatch, 24, (24, 2, 60))
    others = [[1] * 20 + [90, 90], [60, 61, 2, 20, 24, 33] + [0] * 16, [200] + [0] * 21, [9] * 20 + [10, 10]]
    run, state = _scan(kind, first, 16)
    held = _batch([max(n, 1) for n in first])
    held.cu_q = torch.tensor([sum(first[:r]) for r in range(len(first) + 1)], dtype=torch.int32, device=DEV)
    held.q_lens = np.asarray(first, np.int32)
    mine = state.clone()
    run(mine, held)                                         # the library's attributes, the allocator's memory
    mine.copy_(state)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = run(mine, held)
    for lens in others:
        held.cu_q.copy_(torch.tensor([sum(lens[:r]) for r in range(len(lens) + 1)], dtype=torch.int32))
        mine.copy_(state)
        graph.replay()
        want_s, b = state.clone(), _batch([max(n, 1) for n in lens])
        b.cu_q, b.q_lens = held.cu_q, np.asarray(lens, np.int32)
        want = run(want_s, b)
        assert _rel(y, want.double()) < 2e-6 and _rel(mine, want_s.double()) < 2e-6
