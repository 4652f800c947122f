"""The parameter blocks lie one behind the other in a flat buffer, so the bias and the classifier start wherever the embedding
table and the weights end: configurations whose table (vocab x embed) is no multiple of four, or two, floats, and hidden
sizes of every load width, through the fp32 engines against the CPU oracle (the tolerances of the engines' other fp32 tests)."""
import pytest

import oracle
from cavs_b200 import schedule as S
from cavs_b200.treegru import TreeGRU
from cavs_b200.treelstm import TreeLSTM
from helpers import assert_close, make_chain_batch, make_gru_params, make_params, make_tree_batch, tables_from_schedule

pytestmark = pytest.mark.gpu
KEYS = ("state", "loss", "dEmb", "dW", "dU", "dB", "dWc", "dbc")
V = 301


def _batch(seed, batch, K, C):
    if K > 1:
        return make_tree_batch(seed, batch, 2, 14, V, C, max_arity=K)
    parents, tok, label = make_chain_batch(seed, batch, 2, 14, V)
    return parents, tok, label % C


def _check(Engine, reference, params, parents, tok, label, H, E, C, K):
    s = S.Schedule().load(parents, n_slots=K)
    eng = Engine(H, E, V, C, n_slots=K, max_vertices=s.n_total, max_level_rows=s.max_level_rows)
    eng.set_params(params)
    eng.load_batch(s, tok, label)
    eng.forward()
    eng.backward()
    eng.read_loss()
    out = dict(state=eng.state(), loss=eng.loss_rows(), **eng.grad_dict())
    tb = tables_from_schedule(s)
    ref = reference(tb, tok[tb["t2j"]], label[tb["t2j"]], params, H, E, V, C, K=K)
    for k in KEYS:
        assert_close(out[k], ref[k], 1e-5, k, value_tol=4e-5)


@pytest.mark.parametrize("narrow", ["0", "1"])
@pytest.mark.parametrize("H,E,C,K", [
    (100, 50, 5, 2),    # 8-byte offset, hidden a multiple of four
    (100, 25, 5, 3),    # 4-byte offset
    (102, 25, 5, 2),    # 4-byte offset, even hidden size: leaves' gates rebuilt by the backward cell
    (302, 25, 3, 2),    # the same with more than 256 scalars per row
    (64, 25, 10, 1),    # wide loss head: stored d(h) rows
    (33, 22, 4, 2),     # odd hidden size
])
def test_treelstm_fp32(cuda, monkeypatch, H, E, C, K, narrow):
    monkeypatch.setenv("CAVS_NARROW_LEVELS", narrow)
    params = make_params(H, H, E, V, C, scale=0.1, bias_scale=0.05)
    _check(TreeLSTM, oracle.treelstm_fwd_bwd, params, *_batch(900 + H, 11, K, C), H, E, C, K)


@pytest.mark.parametrize("H,E,K", [
    (33, 20, 4),        # odd hidden size: one unit per thread
    (34, 24, 3),        # even: two
    (32, 50, 2),        # multiple of four with the bias on an 8-byte boundary: two
    (32, 25, 2),        # the bias on a 4-byte boundary: one
    (34, 25, 1),
])
def test_treegru_fp32(cuda, H, E, K):
    C = 3
    params = make_gru_params(H, H, E, V, C, scale=0.1, bias_scale=0.05)
    _check(TreeGRU, oracle.treegru_fwd_bwd, params, *_batch(950 + H, 9, K, C), H, E, C, K)
