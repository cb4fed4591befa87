"""The order in which a launch takes a step's sequences, on the CPU, and that their results do not depend on it, on the GPU."""
import numpy as np
import pytest
import torch

from prelude_b200.ops import kernels as K


def _order(lens, counted=True, least=1, n_long=None):
    class Batch:
        q_lens = np.asarray(lens, np.int32)
    return K._longest_first(Batch, K._Split(least, 0, 0, len(lens) if n_long is None else n_long, 0, counted))


@pytest.mark.parametrize("lens", [[5], [592, 1185], [1, 2, 3], [7, 7, 7, 7], [3, 0, 9], list(range(1, 17)), list(range(16, 0, -1)), [4] * 15 + [90]])
def test_longest_first(lens):
    order, longest = _order(lens)
    assert -(1 << 63) <= order < 1 << 63 and longest == max(lens)
    rows = [((order & (1 << 64) - 1) >> 4 * i) & 15 for i in range(len(lens))]
    assert sorted(rows) == list(range(len(lens)))
    assert [lens[r] for r in rows] == sorted(lens, reverse=True)


def test_no_order_where_rows_are_not_the_sequences():
    assert _order([3] * 17) == (0, 0) and _order([3, 4], counted=False) == (0, 0)
    assert _order([3, 4], least=2) == (0, 0) and _order([3, 4], n_long=1) == (0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[70, 300], [65, 1, 200], [10, 20, 30, 40, 50, 60, 70, 80, 90, 100, 110, 120, 130, 140, 150, 160], [66] * 17])
@pytest.mark.parametrize("kind", ["state space", "delta", "gla"])
def test_a_sequence_beside_others_is_what_it_is_alone(kind, lens, monkeypatch):
    """Alone it may be cut into slices of another width, or go token by token: each way is within eight roundings of 6e-8 of 64 bits."""
    import test_gpu_scan_chunks as T
    for name in ("SCAN_CHUNKED_MIN_TOKENS", "DELTA_CHUNKED_MIN_TOKENS", "GLA_CHUNKED_MIN_TOKENS"):
        monkeypatch.setattr(K, name, 1)
    for name in ("SCAN_CHUNKED_LENGTHS", "DELTA_CHUNKED_LENGTHS"):
        monkeypatch.setattr(K, name, (1, 0, 1))
    H, R = 16, len(lens)
    if kind == "state space":
        u, dt, bias, a_log, skip, state = T._ssm_inputs(lens, H, 64, 128, 4, 3, 0.05)

        def run(at, n, s, b):
            return K.ssm_scan(u[at:at + n], dt[at:at + n], bias, a_log, skip, s, b, 4)
    elif kind == "delta":
        u, be, a, a_log, bias, state = T._delta_inputs(lens, H, 8, 128, 128, 3, 0.05)

        def run(at, n, s, b):
            return K.gated_delta_scan(u[at:at + n], be[at:at + n], a[at:at + n], a_log, bias, s, b, 8)
    else:
        q, k, v, decay, state = T._gla_inputs(lens, H, 128, 128, 3, 0.9, 1.0)

        def run(at, n, s, b):
            return K.gla_scan(q[at:at + n], k[at:at + n], v[at:at + n], decay[at:at + n], 0.1, s, b)
    together = state.clone()
    y, at = run(0, sum(lens), together, T._batch(lens)), 0
    for r, n in enumerate(lens):
        alone = state[R - 1 - r:R - r].clone()                      # request r lies in slot R - 1 - r
        one = run(at, n, alone, T._batch([n]))
        for got, want in ((y[at:at + n], one), (together[R - 1 - r], alone[0])):
            assert float((got - want).norm() / want.norm()) < 2 * 8 * 6e-8
        at += n
