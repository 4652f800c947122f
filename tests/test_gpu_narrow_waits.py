"""The bounded waits of the narrow levels' persistent launches, and two engines that use the GPU at once.  With a grid
barrier that never completes its wait runs out (half a second): the launches raise the engine's status word and return with
levels unwritten, whoever takes results to the host gets CAVS_ERR_TIMEOUT, and the context stays usable."""
import threading

import numpy as np
import pytest
import torch

from cavs_b200 import CavsError
from cavs_b200 import schedule as S
from cavs_b200.treelstm import TreeLSTM
from helpers import make_chain_batch, make_params, make_tree_batch

pytestmark = pytest.mark.gpu
CAVS_ERR_TIMEOUT = 4


def _engine(H, E, V, C, K, bf16, parents, tok, label, params):
    s = S.Schedule().load(parents, n_slots=K)
    eng = TreeLSTM(H, E, V, C, n_slots=K, gemm_bf16=bf16, max_vertices=s.n_total, max_level_rows=s.max_level_rows)
    eng.set_params(params)
    eng.load_batch(s, tok, label)
    return eng


def _times_out(call):
    with pytest.raises(CavsError) as e:
        call()
    assert e.value.status == CAVS_ERR_TIMEOUT


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("H,K,C", [(64, 1, 5), (72, 2, 5), (64, 1, 0)])      # C == 0: a layer without a loss head
def test_expired_waits_reach_the_caller(cuda, monkeypatch, bf16, H, K, C):
    E, V = 16, 50
    parents, tok, label = make_chain_batch(5, 6, 2, 9, V) if K == 1 else make_tree_batch(5, 6, 2, 9, V, C)
    label = label % max(C, 1)
    params = make_params(2, H, E, V, max(C, 1))
    args = (H, E, V, C, K, bf16, parents, tok, label if C else None, params)
    monkeypatch.setenv("CAVS_NARROW_WITHHOLD", "1")
    eng = _engine(*args)
    eng.forward()
    for call in (eng.state, eng.check_waits, eng.grad_dict):
        _times_out(call)
    dh = torch.ones((eng.n, H), device=cuda)
    if C == 0:
        eng.set_output_grad(dh)
    eng.backward()
    for call in (eng.read_loss, eng.loss_rows, eng.grad_dict):
        _times_out(call)
    # the same step in the same process without it
    monkeypatch.delenv("CAVS_NARROW_WITHHOLD")
    good = _engine(*args)
    good.forward()
    if C == 0:
        good.set_output_grad(dh)
    good.backward()
    good.check_waits()
    want = dict(state=good.state(), **good.grad_dict())
    assert all(np.isfinite(v).all() for v in want.values()) and np.abs(want["dU"]).max() > 0


@pytest.mark.parametrize("bf16", [False, True])
def test_two_engines_on_two_streams(cuda, bf16):
    # Each thread steps its own engine on its own stream; both keep launching grids that want every SM.
    H, E, V, C, K, steps = 256, 32, 300, 5, 1, 8
    engines, want = [], []
    for i in range(2):
        parents, tok, label = make_chain_batch(40 + i, 30 + 7 * i, 5, 40, V)
        engines.append(_engine(H, E, V, C, K, bf16, parents, tok, label % C, make_params(i, H, E, V, C, scale=0.1, bias_scale=0.05)))
        engines[i].forward()
        engines[i].backward()
        want.append(dict(state=engines[i].state(), **engines[i].grad_dict()))
    torch.cuda.synchronize()

    def work(eng):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(steps):
                eng.grads.zero_()
                eng.forward()
                eng.backward()
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(e,)) for e in engines]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for eng, w in zip(engines, want):
        got = dict(state=eng.state(), **eng.grad_dict())
        for k in w:
            assert np.array_equal(got[k], w[k]), k
