"""Which levels run in the narrow levels' persistent launches is a choice of speed: small widths with levels of thousands of rows
(on both sides of the rule's line) and batches of a few narrow levels give the same results either way.

Tolerance: the engines' tests hold either side to 1e-5 (fp32) and 5e-3 (bf16) of the oracle, so twice that between them."""
import pytest

from cavs_b200 import schedule as S
from cavs_b200.treelstm import TreeLSTM
from helpers import make_chain_batch, make_params, make_tree_batch, rel_err

pytestmark = pytest.mark.gpu
KEYS = ("state", "loss", "dEmb", "dW", "dU", "dB", "dWc", "dbc")


@pytest.mark.parametrize("H,K,batch,hi,bf16", [
    (33, 4, 1500, 6, False),
    (64, 2, 2500, 5, False),
    (32, 1, 3000, 4, False),
    (150, 2, 600, 7, False),
    (512, 1, 250, 12, False),
    (64, 2, 900, 6, True),
    (520, 4, 200, 9, True),
    (1024, 2, 60, 10, True),
    (512, 1, 300, 14, True),
    (1024, 4, 40, 8, True),        # a backward plan but no forward one
])
def test_same_results_either_way(cuda, monkeypatch, H, K, batch, hi, bf16):
    E, V, C = 16, 300, 5
    if K == 1:
        parents, tok, label = make_chain_batch(60 + H, batch, 2, hi, V)
        label %= C
    else:
        parents, tok, label = make_tree_batch(60 + H, batch, 2, hi, V, C, max_arity=K)
    params = make_params(H, H, E, V, C, scale=0.05, bias_scale=0.02)
    s = S.Schedule().load(parents, n_slots=K)
    outs = []
    for narrow in ("0", "1"):
        monkeypatch.setenv("CAVS_NARROW_LEVELS", narrow)
        eng = TreeLSTM(H, E, V, C, n_slots=K, gemm_bf16=bf16, max_vertices=s.n_total, max_level_rows=s.max_level_rows)
        eng.set_params(params)
        eng.load_batch(s, tok, label)
        eng.forward()
        eng.backward()
        outs.append(dict(state=eng.state(), loss=eng.loss_rows(), **eng.grad_dict()))
    for k in KEYS:
        assert rel_err(outs[1][k], outs[0][k]) < (1e-2 if bf16 else 2e-5), k
