"""The work a user of this framework has it do, as cases that can be timed: training steps and forward passes of the
Tree-LSTM, chain-LSTM and Tree-GRU engines through their Python entry points, at the sizes of the benchmark's workloads,
below them and beside them.

A case is a dict of plain values:
    model    "tree" (child-sum Tree-LSTM), "chain" (LSTM language model, `layers` stacked), "gru" (child-sum Tree-GRU)
    mode     "train" (forward + backward, and the update named by `opt`) or "forward"
    batch, lo, hi   samples, and their leaves (trees) or lengths (chains), uniform in lo..hi
    hidden, embed, vocab, classes, slots, bf16
    source   "host": a pass starts from the host's parent / token / label arrays, as a loop over fresh batches does
             (scheduling, table upload, device work); "device": the tables of the batch are resident, as in an engine
             whose batches are staged beside the step
    opt      "none" (gradients), "sgd", "adagrad"
    sparse   the loader lists the embedding rows that the batch touches (compact embedding-gradient block)
"""
from __future__ import annotations

import numpy as np
import torch

from cavs_b200 import schedule as S
from cavs_b200.treegru import TreeGRU
from cavs_b200.treelstm import TreeLSTM

_LR = {"sgd": 1.0, "adagrad": 0.05, "none": 0.0}


def _case(name, model, mode, batch, lo, hi, hidden, embed, vocab, classes, slots, bf16, source, opt="none", sparse=False, layers=1, scale=0.05):
    return dict(name=name, model=model, mode=mode, batch=batch, lo=lo, hi=hi, hidden=hidden, embed=embed, vocab=vocab, classes=classes,
                slots=slots, bf16=bf16, source=source, opt=opt, sparse=sparse, layers=layers, scale=scale)


def listed():
    return [
        # One sentence through a trained sentiment classifier: the latency of a single request, host to host.
        _case("tree_forward_1", "tree", "forward", 1, 20, 50, 150, 300, 21701, 5, 2, False, "host"),
        # The sentiment-treebank training step in fp32: 64 trees per step, a loss on every vertex, Adagrad.
        _case("tree_train_64", "tree", "train", 64, 2, 50, 150, 300, 21701, 5, 2, False, "host", "adagrad"),
        # The small language model: fixed length 20, batch 20, vocabulary-sized softmax, SGD with learning rate 1.
        _case("chain_train_20", "chain", "train", 20, 20, 20, 200, 200, 10000, 10000, 1, False, "host", "sgd", scale=0.1),
        # Two stacked LSTM layers over ragged sequences, fp32, vocabulary-sized softmax.
        _case("chain2_train_256", "chain", "train", 256, 10, 100, 512, 512, 10000, 10000, 1, False, "device", layers=2),
        # The same model with bf16 products on a smaller batch of shorter sequences.
        _case("chain2_train_bf16_96", "chain", "train", 96, 5, 60, 512, 512, 10000, 10000, 1, True, "device", layers=2),
        # N-ary Tree-GRU, bf16 products, one label per tree.
        _case("gru_train_512", "gru", "train", 512, 8, 128, 1024, 512, 32000, 2, 4, True, "device"),
        # Four-ary Tree-LSTM with a width that is no multiple of the tensor cores' tile and an odd batch, fresh batches.
        _case("tree_train_4ary_301", "tree", "train", 301, 3, 77, 520, 264, 21701, 3, 4, True, "host", "adagrad"),
        # One rank's shard of the large data-parallel configuration on eight GPUs: deep, narrow levels.
        _case("tree_train_512", "tree", "train", 512, 2, 128, 1024, 1024, 50000, 5, 2, True, "device", "adagrad"),
        # Evaluation pass at that width: states of every vertex, no gradients.
        _case("tree_forward_1024", "tree", "forward", 1024, 2, 128, 1024, 1024, 50000, 5, 2, True, "device"),
        # The large configuration on one GPU, with the touched embedding rows listed by the loader.
        _case("tree_train_4096", "tree", "train", 4096, 2, 128, 1024, 1024, 50000, 5, 2, True, "device", "adagrad", True),
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of lo..hi."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["tree_f32", "tree_f32", "tree_bf16", "tree_bf16", "tree_bf16", "chain_f32", "chain_bf16", "gru"])
    source = rng.choice(["host", "device"])
    if kind == "tree_f32":
        # treebank-sized classifiers; any hidden size
        mode = rng.choice(["train", "train", "forward"])
        slots = rng.choice([2, 2, 3, 4]) if mode == "train" else 2
        c = _case("", "tree", mode, _log(rng, 1, 256), 2, _log(rng, 4, 64), _log(rng, 32, 320), 4 * _log(rng, 8, 100), _log(rng, 1000, 50000),
                  rng.randint(2, 8), slots, False, source, rng.choice(["adagrad", "sgd"]) if mode == "train" else "none")
    elif kind == "tree_bf16":
        mode = rng.choice(["train", "train", "train", "forward"])
        slots = rng.choice([2, 2, 3, 4]) if mode == "train" else 2
        c = _case("", "tree", mode, _log(rng, 16, 2048), 2, _log(rng, 8, 128), 8 * _log(rng, 32, 128), 8 * _log(rng, 16, 128), _log(rng, 5000, 50000),
                  rng.randint(2, 8), slots, True, source if mode == "train" else "device", "adagrad" if mode == "train" else "none", mode == "train" and rng.random() < 0.5)
    elif kind == "chain_f32":
        v = _log(rng, 1000, 10000)
        h = 4 * _log(rng, 16, 128)
        c = _case("", "chain", "train", _log(rng, 8, 256), 2, _log(rng, 10, 100), h, h, v, v, 1, False, source, rng.choice(["none", "sgd"]),
                  layers=rng.choice([1, 2]))
    elif kind == "chain_bf16":
        v = 8 * _log(rng, 125, 1250)
        h = 8 * _log(rng, 16, 128)
        c = _case("", "chain", "train", _log(rng, 8, 256), 2, _log(rng, 10, 100), h, h, v, v, 1, True, source, rng.choice(["none", "sgd"]),
                  layers=rng.choice([1, 2]))
    else:
        bf16 = rng.random() < 0.75
        c = _case("", "gru", "train", _log(rng, 16, 512) if bf16 else _log(rng, 4, 64), 2, _log(rng, 8, 128), 8 * _log(rng, 32, 128) if bf16 else 2 * _log(rng, 16, 150),
                  8 * _log(rng, 16, 128), _log(rng, 5000, 32000), rng.randint(2, 8), rng.choice([2, 3, 4]), bf16, source)
    del c["name"]
    return c


def _batch(case, seed):
    """Parent, token and label arrays of one batch: tokens Zipf(1.1) on the leaves (trees) or on every vertex (chains)."""
    seed = seed * 1000003
    if case["model"] == "chain":
        parents = S.synth_chains(seed, case["batch"], case["lo"], case["hi"])
        is_word = None
    elif case["mode"] == "forward":
        # binary trees whose leaf counts belong to the case and whose shapes are the seed's: as many states for every seed
        leaves = np.random.default_rng([case["batch"], case["lo"], case["hi"]]).integers(case["lo"], case["hi"] + 1, case["batch"])
        parents = np.full((case["batch"], 2 * case["hi"] - 1), -1, np.int32)
        is_word = np.zeros(parents.shape, np.uint8)
        for i, k in enumerate(leaves):
            p, w = S.synth_trees(seed + 3 + i, 1, int(k), int(k))
            parents[i, :p.shape[1]], is_word[i, :p.shape[1]] = p[0], w[0]
    else:
        parents, is_word = S.synth_trees(seed, case["batch"], case["lo"], case["hi"], case["slots"])
    lens = (parents == -1).argmax(1) + 1
    mask = np.arange(parents.shape[1])[None, :] < lens[:, None]
    tok = S.synth_zipf(seed + 1, 1.1, case["vocab"], parents.size).reshape(parents.shape)
    tok = np.ascontiguousarray((tok if is_word is None else tok * is_word)[mask], np.int32)
    n = tok.size
    last = np.cumsum(lens) - 1
    if case["model"] == "chain":        # the next token; the last position predicts token 0
        label = np.zeros(n, np.int32)
        label[:-1] = tok[1:]
        label[last] = 0
    elif case["model"] == "gru":        # one label per tree, on its root
        label = np.full(n, -1, np.int32)
        label[last] = S.synth_uniform_int(seed + 2, case["classes"], case["batch"])
    else:
        label = S.synth_uniform_int(seed + 2, case["classes"], n)
    return parents, tok, label


def _engines(case, n, rows, seed):
    H, E, V, C = case["hidden"], case["embed"], case["vocab"], case["classes"]
    cap = dict(n_slots=case["slots"], gemm_bf16=case["bf16"], max_vertices=n, max_level_rows=rows)
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    if case["model"] == "gru":
        eng = TreeGRU(H, E, V, C, **cap)
        shapes = dict(Emb=V * E, W=3 * E * H, U=3 * H * H, B=3 * H, Wc=C * H, bc=C)
        draws = {k: torch.empty(s, device="cuda").uniform_(-case["scale"], case["scale"], generator=gen).cpu().numpy() for k, s in shapes.items()}
        eng.set_params(draws)
        return [eng]
    engines = []
    for layer in range(case["layers"]):
        eng = TreeLSTM(H, E if layer == 0 else H, V if layer == 0 else 0, C if layer == case["layers"] - 1 else 0, **cap)
        eng.params.uniform_(-case["scale"], case["scale"], generator=gen)
        eng.refresh_weights()
        engines.append(eng)
    return engines


def prepare(case, seed):
    parents, tok, label = _batch(case, seed)
    sched = S.Schedule().load(parents, n_slots=case["slots"])
    engines = _engines(case, sched.n_total, sched.max_level_rows, seed)
    state = dict(case=case, parents=parents, tok=tok, label=label, sched=sched, engines=engines)
    state["loss_rows"] = case["batch"] if case["model"] == "gru" else sched.n_total
    state["rows"] = np.unique(tok) if case["sparse"] else None
    if case["opt"] == "adagrad":
        # an accumulator as it is in the middle of training: the update is then a smooth function of the gradient
        state["acc"] = torch.full_like(engines[0].params, 0.1)
    if case["source"] == "device":
        _load(state)
    return state


def _load(state):
    """The batch's schedule becomes the engines' current one: packing and upload of its tables."""
    engines, sched, rows = state["engines"], state["sched"], state["loss_rows"]
    if state["case"]["model"] == "gru":
        engines[0].load_batch(sched, state["tok"], state["label"], loss_rows=rows)
        return
    for i, eng in enumerate(engines):
        eng.load_batch(sched, state["tok"] if i == 0 else None, state["label"] if i == len(engines) - 1 else None, loss_rows=rows,
                       exchange_rows=state["rows"])


def _layers_pass(engines, n):
    """Forward bottom-up (a layer's h columns feed the next layer), backward top-down."""
    H = engines[0].cfg.hidden
    for i, eng in enumerate(engines):
        if i > 0:
            eng.set_dense_input(engines[i - 1].device_view(0, (n, 2 * H))[:, :H])
        eng.forward()
    for i in range(len(engines) - 1, -1, -1):
        if i < len(engines) - 1:
            engines[i].set_output_grad(engines[i + 1].device_view(5, (n, H)))
        engines[i].backward()


def run(state):
    case, engines, sched = state["case"], state["engines"], state["sched"]
    eng = engines[0]
    if case["source"] == "host":
        if case["model"] == "tree" and case["mode"] == "train":
            eng.stage(sched, state["parents"], state["tok"], state["label"], loss_rows=state["loss_rows"], exchange_rows=state["rows"])
        else:
            sched.load(state["parents"], n_slots=case["slots"])
            _load(state)
    n = sched.n_total
    if case["mode"] == "forward":
        eng.forward()
        if case["source"] == "host":
            return {"state": eng.state()}                       # a request's answer goes back to the host
        H, leaves = case["hidden"], int(sched.level_off[1])
        return {"state": eng.device_view(0, (n, 2 * H))[leaves:]}   # states of the internal vertices, for what follows on the GPU
    if case["model"] == "gru":
        eng.forward()
        eng.backward()
        return {"grads": eng.grads}
    if case["model"] == "chain":
        _layers_pass(engines, n)
        if case["opt"] == "sgd":
            for e in engines:
                e.sgd(_LR["sgd"])
    else:
        opt = {"none": eng.OPT_NONE, "sgd": eng.OPT_SGD, "adagrad": eng.OPT_ADAGRAD}[case["opt"]]
        eng.step(None, opt, state.get("acc"), _LR[case["opt"]])
    out = {"loss": engines[-1].device_view(6, (2,))[:1]}
    for i, e in enumerate(engines):
        for k in e.PARAM_NAMES:
            if e.sizes[k]:
                g = e.view(e.grads, k)
                if k != "Emb" or state["rows"] is None:
                    out[f"d{k}{i}"] = g
                else:                           # one gradient row per listed table row: what it did to the optimizer's state
                    out["acc0"] = e.view(state["acc"], k)
        if case["opt"] != "none":
            out[f"params{i}"] = e.params
    return out


def work(case):
    """Bytes: parameters, batch arrays, optimizer state in; gradients, updated parameters, states out.  Flops: the products
    with the input weights once per distinct token, with the recurrent weights once per vertex that has children (per
    distinct token where all children are leaves with tokens), with a vocabulary-sized classifier once per vertex."""
    parents, tok, label = _batch(case, 0)
    sched = S.Schedule().load(parents, n_slots=case["slots"])
    H, E, V, C, n = case["hidden"], case["embed"], case["vocab"], case["classes"], sched.n_total
    off = sched.level_off
    child = sched.adjacency()[1]
    tokens = len(np.unique(tok))
    n_int = n - int(off[1])
    links = int((child >= 0).sum())
    n_top = n_int - (int(off[2] - off[1]) if len(off) > 2 and case["model"] == "tree" else 0)   # vertices above level 1
    links_top = links * n_top // max(n_int, 1)
    gates = 3 if case["model"] == "gru" else 4
    train = case["mode"] == "train"
    times = 3.0 if train else 1.0
    flops, bytes_ = 0.0, 4.0 * (parents.size + 2 * n)
    for layer in range(case["layers"]):
        rows_in = tokens if layer == 0 else n
        e_in = E if layer == 0 else H
        flops += times * 2.0 * rows_in * e_in * gates * H
        if case["model"] == "gru":
            flops += times * 2.0 * H * H * (2 * n_int + links)
        else:
            flops += times * 2.0 * H * H * (3 * n_top + links_top + (4 * tokens if n_top < n_int else 0))
        weights = 4.0 * (e_in * gates * H + gates * H * H + gates * H)
        if train:
            bytes_ += 2 * weights + (8.0 * tokens * E if layer == 0 else 0.0)   # weights in, gradients out
            if case["opt"] != "none":
                bytes_ += weights + (4.0 * tokens * E if layer == 0 else 0.0)
                if case["opt"] == "adagrad":
                    bytes_ += 2 * weights + (8.0 * tokens * E if layer == 0 else 0.0)
            if layer == 0 and not case["sparse"]:
                bytes_ += 4.0 * (V - tokens) * E                                 # the untouched rows of the dense gradient block
        else:
            bytes_ += weights + (4.0 * tokens * E if layer == 0 else 0.0) + 8.0 * H * (n if case["source"] == "host" else n_int)
    if train:
        head_rows = n if case["model"] != "gru" else case["batch"]
        flops += 3.0 * 2.0 * head_rows * H * C
        bytes_ += 8.0 * C * H
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Four times what was measured against the same step in 64 bits (and no less than 1e-5 in fp32): bf16 products 4.7e-3
    (2-norm); fp32 1e-6, but 5.4e-5 in a vocabulary-sized classifier's gradient summed over 14,474 rows (9e-7 over 3,000).
    The largest single difference, relative to an embedding gradient's mean square over all its rows, most of them zero,
    was 0.65 with bf16 products."""
    if case["bf16"]:
        return {"rel": 0.02, "max": 0.99}
    rows = case["batch"] * (case["lo"] + case["hi"]) / 2 if case["model"] == "chain" else 0
    rel = 1e-5 + 1.5e-8 * rows
    return {"rel": rel, "max": 40 * rel}
