"""What users of this framework have it do, as timed cases.

A case is a dict of plain values; its ``mode`` says which public entry point it goes through:

* ``act``    one acting step of a vectorised environment loop: ``Memoroid(cell)`` on (B, 1, F), no gradients, the carry
             of the last step threaded into the next;
* ``scan``   the bare real recurrence, ``ops.linrec_fwd`` (a host that owns its own cell);
* ``infer``  a forward pass over whole segments without gradients (values of a rollout, evaluation);
* ``train``  a layer in a policy or value update: forward over a segment with resets, then the gradients of the
             inputs and of every parameter from the cotangent of the outputs;
* ``rtrl``   one real-time-recurrent-learning segment, ``Memoroid.local_jacobian`` with the LRU cell;
* ``step``   one whole training step (forward, backward, Adam) of the four-layer value network.

The log-domain, complex and Mamba cells run in float32, the attention-style cells in bfloat16, which is how the
benchmark and the tests run them."""
import math

import torch

from memorax_b200 import ops
from memorax_b200.blocks import FlatAdamTrainer, GTrXLStyleValueNet
from memorax_b200.memoroid import (DeltaNetCell, LinearAttentionCell, LRUCell, MambaCell, Memoroid, MinGRUCell,
                                   mLSTMCell)

#: cells whose modules and activations are bfloat16; the others are float32
BF16_CELLS = ("linattn", "deltanet", "mlstm")
#: share of the steps that begin a new episode
P_DONE = 0.01


def listed():
    return [
        # the smallest call: sixteen environments take one step (the inner loop of every on-policy rollout)
        {"name": "act-lru", "mode": "act", "cell": "lru", "batch": 16, "features": 128, "hidden": 256},
        # a wide vectorised environment with an attention-style memory: the (B, H, d, d) state goes in and out
        {"name": "act-linattn", "mode": "act", "cell": "linattn", "batch": 256, "features": 256, "heads": 4, "head_dim": 64},
        # benchmark configuration 1: the real recurrence on a short segment, forward only
        {"name": "scan-real", "mode": "scan", "batch": 64, "steps": 128, "features": 256},
        # benchmark row n4: the LRU layer over a large rollout, the largest forward-only call
        {"name": "infer-lru", "mode": "infer", "cell": "lru", "batch": 1024, "steps": 1024, "features": 256, "hidden": 512,
         "carry": False},
        # the LRU layer (benchmark configuration 4's recurrence, 512 states) in an update over 256 sequences
        {"name": "train-lru", "mode": "train", "cell": "lru", "batch": 256, "steps": 256, "features": 256, "hidden": 512,
         "carry": True},
        # MinGRU in an update; sequence count and length as they come out of a minibatch split, not powers of two
        {"name": "train-mingru", "mode": "train", "cell": "mingru", "batch": 96, "steps": 250, "features": 512, "carry": True},
        # the layer around benchmark configuration 2 (4 heads of 64, 256 x 256)
        {"name": "train-linattn", "mode": "train", "cell": "linattn", "batch": 256, "steps": 256, "features": 256, "heads": 4,
         "head_dim": 64, "carry": True},
        # the layer around benchmark configuration 3 (8 heads of 128, 128 x 512)
        {"name": "train-deltanet", "mode": "train", "cell": "deltanet", "batch": 128, "steps": 512, "features": 512, "heads": 8,
         "head_dim": 128, "carry": False},
        # the shipped example's Mamba layer: 512 features, 8 heads of 16 x 16, 128 environments x 64 steps
        {"name": "train-mamba", "mode": "train", "cell": "mamba", "batch": 128, "steps": 64, "features": 512, "heads": 8,
         "head_dim": 16, "state_dim": 16, "carry": True},
        # mLSTM on the tensor cores, a ragged minibatch
        {"name": "train-mlstm", "mode": "train", "cell": "mlstm", "batch": 60, "steps": 100, "features": 256, "heads": 4,
         "head_dim": 64, "carry": True},
        # benchmark row n3: an RTRL segment of the LRU cell
        {"name": "rtrl-lru", "mode": "rtrl", "batch": 64, "steps": 64, "features": 64, "hidden": 128},
        # benchmark configuration 5 on one GPU: 512 sequences x 256 steps of 128-dimensional observations
        {"name": "step-gtrxl", "mode": "step", "batch": 512, "steps": 256},
    ]


def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _cell_sizes(rng, cell):
    if cell == "lru":
        return {"features": rng.choice((64, 96, 128, 192, 256)), "hidden": rng.choice((64, 128, 200, 256, 384, 512))}
    if cell == "mingru":
        return {"features": rng.choice((64, 128, 192, 256, 384, 512))}
    if cell == "mamba":
        return {"features": rng.choice((128, 256, 384, 512)), "heads": rng.choice((4, 8)), "head_dim": 16, "state_dim": 16}
    if cell == "deltanet":
        return {"features": rng.choice((256, 512)), "heads": rng.choice((2, 4, 8)), "head_dim": rng.choice((64, 128))}
    return {"features": rng.choice((128, 256, 512)), "heads": rng.choice((2, 4, 8)), "head_dim": rng.choice((32, 64))}


def draw(rng):
    mode = rng.choice(("act", "act", "scan", "infer", "train", "train", "train", "train", "rtrl", "step"))
    if mode == "act":
        cell = rng.choice(("lru", "mingru", "linattn", "deltanet"))
        return {"mode": mode, "cell": cell, "batch": _log(rng, 1, 1024), **_cell_sizes(rng, cell)}
    if mode == "scan":
        return {"mode": mode, "batch": _log(rng, 1, 256), "steps": _log(rng, 16, 1024), "features": 4 * _log(rng, 8, 256)}
    if mode == "infer":
        cell = rng.choice(("lru", "mingru", "linattn"))
        steps = _log(rng, 16, 1024)
        return {"mode": mode, "cell": cell, "batch": _log(rng, 8, min(1024, 262144 // steps)), "steps": steps,
                **_cell_sizes(rng, cell), "carry": rng.random() < 0.5}
    if mode == "train":
        cell = rng.choice(("lru", "mingru", "linattn", "deltanet", "mamba", "mlstm"))
        steps = _log(rng, 16, 512)
        return {"mode": mode, "cell": cell, "batch": _log(rng, 8, min(256, 65536 // steps)), "steps": steps,
                **_cell_sizes(rng, cell), "carry": rng.random() < 0.5}
    if mode == "rtrl":
        return {"mode": mode, "batch": _log(rng, 8, 128), "steps": _log(rng, 8, 128), "features": rng.choice((16, 32, 64, 128)),
                "hidden": rng.choice((32, 64, 128, 256))}
    return {"mode": mode, "batch": _log(rng, 8, 512), "steps": _log(rng, 32, 256)}


def _model(case):
    """The layer with weights as its initialisers draw them (from the global generator), on the GPU."""
    cell = case["cell"]
    with torch.device("cuda"):
        if cell == "lru":
            made = LRUCell(case["features"], case["hidden"], r_min=0.9, r_max=0.999, max_phase=math.pi / 10)
        elif cell == "mingru":
            made = MinGRUCell(case["features"])
        elif cell == "mamba":
            made = MambaCell(case["features"], num_heads=case["heads"], head_dim=case["head_dim"], state_dim=case["state_dim"])
        elif cell == "linattn":
            made = LinearAttentionCell(case["features"], case["head_dim"], case["heads"])
        elif cell == "deltanet":
            made = DeltaNetCell(case["features"], case["head_dim"], case["heads"])
        else:
            made = mLSTMCell(case["features"], case["heads"] * case["head_dim"], num_heads=case["heads"], tensor_cores=True)
            with torch.no_grad():     # the gates start at zero weights; a layer in training has left that point
                made.i_gate.weight.normal_(std=0.02)
                made.f_gate.weight.normal_(std=0.02)
    model = Memoroid(made)
    return model.to(torch.bfloat16) if cell in BF16_CELLS else model


def _carry(case, gen):
    """A carry as an earlier segment leaves it, in the layout of ``initialize_carry``."""
    b = case["batch"]
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    cell = case["cell"]
    if cell == "lru":
        state = torch.view_as_complex(rn(b, 1, case["hidden"], 2))
        return state, torch.ones_like(state)
    if cell == "mingru":
        return rn(b, 1, case["features"]), -rn(b, 1, case["features"]).abs()
    if cell == "mamba":
        shape = (b, 1, case["heads"], case["state_dim"], case["head_dim"])
        return 0.1 * rn(*shape), torch.rand(b, 1, case["heads"], 1, 1, generator=gen, device="cuda")
    h, d = case["heads"], case["head_dim"]
    if cell == "linattn":
        return 0.1 * rn(b, 1, h, d, d), 0.1 * rn(b, 1, h, d).abs()
    if cell == "deltanet":
        return (0.1 * rn(b, 1, h, d, d),)
    return 0.1 * rn(b, 1, h, d, d), -rn(b, 1, h, 1, 1).abs(), 0.1 * rn(b, 1, h, d, 1), 0.1 * rn(b, 1, h, 1, 1)


def prepare(case, seed):
    mode, b = case["mode"], case["batch"]
    steps = case.get("steps", 1)
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    state = {"mode": mode, "done": torch.rand(b, steps, generator=gen, device="cuda") < P_DONE}
    if mode == "scan":
        shape = (b, steps, case["features"])
        return dict(state, a=torch.sigmoid(rn(*shape)), b=rn(*shape), h0=rn(b, case["features"]))
    if mode == "step":
        with torch.device("cuda"):
            net = GTrXLStyleValueNet().to(torch.bfloat16)
        return dict(state, trainer=FlatAdamTrainer(net), obs=rn(b, steps, 128).bfloat16(), target=rn(b, steps))
    if mode == "rtrl":
        model = _model(dict(case, cell="lru"))
        c64 = lambda t: 0.1 * torch.view_as_complex(rn(*t.shape, 2))
        sens = {k: c64(v) for k, v in model.initialize_sensitivity(None, (b, case["features"])).items()}
        return dict(state, model=model, x=rn(b, steps, case["features"]), carry=_carry(dict(case, cell="lru"), gen), sens=sens)
    dtype = torch.bfloat16 if case["cell"] in BF16_CELLS else torch.float32
    model = _model(case)
    state.update(model=model, x=rn(b, steps, case["features"]).to(dtype),
                 carry=_carry(case, gen) if mode == "act" or case["carry"] else None)
    if mode == "train":
        state["x"].requires_grad_()
        state.update(wrt=[state["x"], *model.parameters()], gy=rn(b, steps, case["features"]).to(dtype))
    return state


def run(state):
    mode = state["mode"]
    if mode == "scan":
        return ops.linrec_fwd(state["a"], state["b"], state["h0"], None, state["done"])
    if mode == "step":
        trainer = state["trainer"]
        loss = trainer.step(state["obs"], state["done"], state["target"])
        return loss, trainer.flat, trainer.flat_grad, trainer.master, trainer.m, trainer.v
    if mode == "rtrl":
        with torch.no_grad():
            return state["model"].local_jacobian(state["x"], state["done"], state["carry"], state["sens"])
    if mode == "train":
        carry, y = state["model"](state["x"], state["done"], state["carry"])
        grads = torch.autograd.grad(y, state["wrt"], state["gy"])
        return carry, y, grads
    with torch.no_grad():
        carry, y = state["model"](state["x"], state["done"], state["carry"])
    if mode == "act":
        state["carry"] = carry
    return carry, y


def _layer(case):
    """(weights, carry elements in float32 words, flops of the mixing per token, bytes of an activation) of a layer."""
    f, cell = case["features"], case["cell"]
    if cell == "lru":
        n = case["hidden"]
        return 4 * n * f + 3 * n + f, 4 * n, 8 * n, 4
    if cell == "mingru":
        return 2 * f * f, 2 * f, 20 * f, 4
    h, d = case["heads"], case["head_dim"]
    if cell == "mamba":
        n = case["state_dim"]
        return f * (2 * h * d + 2 * h * n + h) + 5 * (h * d + 2 * h * n) + h * d * (f + 1) + f, h * (n * d + 1), 4 * h * n * d, 4
    if cell == "linattn":
        return 4 * f * h * d + h * d + f, h * d * (d + 1), 4 * h * d * d, 2
    if cell == "deltanet":
        return 4 * f * h * d + 2 * h * (f + 1) + h * d + f, h * d * d, 6 * h * d * d, 2
    e = h * d
    return 3 * f * e + 3 * h * d * d + 6 * h * e + 8 * e, h * (d * d + d + 2), 4 * h * d * d, 2


def work(case):
    b, steps = case["batch"], case.get("steps", 1)
    tokens = b * steps
    if case["mode"] == "scan":
        n = tokens * case["features"]
        return {"bytes": 12 * n + tokens + 8 * b * case["features"], "flops": 2 * n}
    if case["mode"] == "rtrl":
        f, n = case["features"], case["hidden"]
        sens = b * n * (3 + 2 * f)
        return {"bytes": 8 * tokens * f + 4 * (4 * n * f + 3 * n + f) + 16 * sens + 32 * b * n + tokens,
                "flops": 8 * tokens * n * f + 8 * tokens * n * (4 + 2 * f)}
    if case["mode"] == "step":
        dense = 128 * 512 + 512 + 4 * (512 * 512 * 6 + 512 * 16 + 8 * 512 * 512)
        # parameters, gradients and both moments once each way; observations and targets in
        return {"bytes": 32 * dense + tokens * (128 * 2 + 4 + 1), "flops": tokens * (6 * dense + 4 * 18 * 8 * 64 * 64)}
    weights, carry, mixing, size = _layer(case)
    passes = 3 if case["mode"] == "train" else 1
    # forward: inputs in, outputs out; with gradients also the outputs' cotangent in, the inputs' and weights' out
    acts = tokens * case["features"] * size * (4 if passes == 3 else 2)
    carries = 4 * b * carry * (2 if case["mode"] == "act" or case["carry"] else 1)
    return {"bytes": acts + weights * size * (2 if passes == 3 else 1) + carries + tokens,
            "flops": passes * tokens * (2 * weights + mixing)}


def tolerance(case):
    if case["mode"] == "step":
        return {"rel": 2e-2}      # bfloat16 through four layers and back; the second moment is a square
    if case.get("cell") in BF16_CELLS:
        return {"rel": 2e-2 if case["mode"] == "train" else 1e-2}
    # float32: gradients of parameters are sums over every step of every sequence
    return {"rel": 5e-5 if case["mode"] == "train" else 1e-5}
