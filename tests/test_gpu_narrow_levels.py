"""The narrow levels of the Tree-LSTM (one persistent launch per direction) against the CPU oracle.  fp32: hidden sizes of
every load width (odd, even, multiples of four), gate-gradient rows that fit the shared-memory buffers at once and ones
that do not, one to four child slots, partial row tiles, levels on both sides of the plan's split.  bf16: hidden sizes
with and without the gate epilogue's layout of the saved gates, k ranges that do not divide over the warps, gradient rows
that fit the buffers and ones that do not."""
import numpy as np
import pytest

import oracle
from cavs_b200 import schedule as S
from cavs_b200.treelstm import TreeLSTM
from helpers import assert_close, make_params, make_tree_batch, rel_err, tables_from_schedule

pytestmark = pytest.mark.gpu
KEYS = ("state", "loss", "dEmb", "dW", "dU", "dB", "dWc", "dbc")


@pytest.mark.parametrize("H,K,batch,hi,C", [
    (33, 2, 40, 12, 5),       # odd width: scalar loads
    (150, 2, 130, 6, 5),      # pairs; levels above and below 96 rows
    (150, 4, 20, 20, 3),
    (320, 2, 3, 30, 5),       # two rounds of buffers
    (512, 1, 33, 40, 5),      # one child slot, rows just over a tile
    (512, 1, 150, 9, 5),      # wide levels first, then narrow ones
    (152, 3, 30, 15, 8),
    (7, 1, 1, 60, 2),         # fewer units than a column group
])
def test_parity_with_oracle(cuda, H, K, batch, hi, C):
    E, V = 20, 300
    if K == 1:
        parents = S.synth_chains(500 + H, batch, 2, hi)
        lens = (parents == -1).argmax(1) + 1
        tok = S.synth_zipf(6, 1.1, V, int(lens.sum()))
        label = S.synth_uniform_int(7, C, int(lens.sum()))
    else:
        parents, tok, label = make_tree_batch(500 + H + K, batch, 2, hi, V, C, max_arity=K)
    params = make_params(H, H, E, V, C, scale=0.1, bias_scale=0.05)
    s = S.Schedule().load(parents, n_slots=K)
    eng = TreeLSTM(H, E, V, C, n_slots=K, max_vertices=s.n_total, max_level_rows=s.max_level_rows)
    eng.set_params(params)
    eng.load_batch(s, tok, label)
    outs = []
    for _ in range(2):
        eng.forward()
        eng.backward()
        eng.read_loss()                   # raises if a bounded wait ran out
        outs.append(dict(state=eng.state(), loss=eng.loss_rows(), **eng.grad_dict()))
    tb = tables_from_schedule(s)
    ref = oracle.treelstm_fwd_bwd(tb, tok[tb["t2j"]], label[tb["t2j"]], params, H, E, V, C, K=K)
    for k in KEYS:
        assert_close(outs[0][k], ref[k], 1e-5, k, value_tol=4e-5)
        assert np.array_equal(outs[0][k], outs[1][k]), k       # deterministic


@pytest.mark.parametrize("H,K,batch,hi", [
    (64, 2, 30, 16),          # one k step for each of four warps
    (200, 2, 20, 30),         # 12.5 k steps; saved gates in one array
    (512, 1, 70, 30),         # row tiles of 32, the last one partial
    (520, 4, 12, 12),
    (1024, 2, 9, 24),         # fewer buffers than vectors
    (256, 3, 25, 10),
])
def test_bf16_parity_with_oracle(cuda, monkeypatch, H, K, batch, hi):
    E, V, C = 24, 300, 5
    if K == 1:
        parents = S.synth_chains(700 + H, batch, 2, hi)
        lens = (parents == -1).argmax(1) + 1
        tok = S.synth_zipf(6, 1.1, V, int(lens.sum()))
        label = S.synth_uniform_int(7, C, int(lens.sum()))
    else:
        parents, tok, label = make_tree_batch(700 + H + K, batch, 2, hi, V, C, max_arity=min(K, 4))
    params = make_params(H, H, E, V, C, scale=0.05, bias_scale=0.02)
    s = S.Schedule().load(parents, n_slots=K)
    tb = tables_from_schedule(s)
    ref = oracle.treelstm_fwd_bwd(tb, tok[tb["t2j"]], label[tb["t2j"]], params, H, E, V, C, K=K, gemm_bf16=True, preact_bf16=True)
    outs = {}
    for narrow in ("1", "1", "0"):
        monkeypatch.setenv("CAVS_NARROW_LEVELS", narrow)
        eng = TreeLSTM(H, E, V, C, n_slots=K, gemm_bf16=True, max_vertices=s.n_total, max_level_rows=s.max_level_rows)
        eng.set_params(params)
        eng.load_batch(s, tok, label)
        eng.forward()
        eng.backward()
        eng.read_loss()                   # raises if a bounded wait ran out
        out = dict(state=eng.state(), loss=eng.loss_rows(), **eng.grad_dict())
        for k in KEYS:
            assert rel_err(out[k], ref[k]) < 5e-3, (narrow, k)      # same rounding points as the oracle's bf16 mode
            if narrow in outs:
                assert np.array_equal(out[k], outs[narrow][k]), k    # deterministic
        outs[narrow] = out
