"""Workloads of the pair-stack operators, as a program that uses this package runs them.

Every case is one call a model makes on a pair tensor ``z [B, N, N, C]``: a triangle multiplicative update (outgoing,
incoming or both directions in one operator) or the pair Transition, either as an inference forward (bf16 parameters, no
graph) or as a training step (forward and backward with fp32 master weights; output, input gradient and every parameter
gradient come back). The keys of a case:

  op     "outgoing", "incoming", "bidirectional" (the three triangle updates) or "transition"
  mode   "infer" or "train"
  c      channels of the pair tensor: 128, or 64 for the narrow stacks (template blocks, small trunks)
  b, n   samples and tokens
  mask   "none", "token" ([B, N]) or "pair" ([B, N, N])
  drop   True: the training forward applies the row-shared dropout (p = 0.25) with a given scale
"""

import math

import torch
import torch.nn.functional as F

import miniworld_b200 as mw
from miniworld_b200.training import trimul_train

TRIMUL = ("outgoing", "incoming", "bidirectional")


def _case(name, op, mode, c, b, n, mask="token", drop=False):
    case = {"op": op, "mode": mode, "c": c, "b": b, "n": n, "mask": mask, "drop": drop}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # a peptide or a small ligand complex: the call is launches and latency
        _case("infer_out_n64", "outgoing", "infer", 128, 1, 64),
        # a protein of ordinary length served as it is, without padding the sequence to a round number
        _case("infer_in_n203", "incoming", "infer", 128, 1, 203, mask="pair"),
        # a 384-token crop, the reference's usual benchmark length
        _case("infer_out_n384", "outgoing", "infer", 128, 1, 384),
        # a 768-token crop, the benchmark's headline length
        _case("infer_in_n768", "incoming", "infer", 128, 1, 768),
        # a batch of short proteins of different lengths, padded at the end
        _case("infer_out_b8_n256", "outgoing", "infer", 128, 8, 256),
        # a large complex
        _case("infer_in_n2048", "incoming", "infer", 128, 1, 2048),
        # the one operator that the reference's own trunk builds
        _case("infer_bidir_n512", "bidirectional", "infer", 128, 1, 512),
        # four templates in a 64-wide template stack
        _case("infer_narrow_b4_n256", "outgoing", "infer", 64, 4, 256),
        # the feed-forward that follows every triangle update
        _case("infer_transition_n512", "transition", "infer", 128, 1, 512, mask="none"),
        # training on crops: the triangle update, the trunk's operator with dropout, the feed-forward
        _case("train_out_n384", "outgoing", "train", 128, 1, 384),
        _case("train_bidir_drop_n256", "bidirectional", "train", 128, 1, 256, drop=True),
        _case("train_transition_n384", "transition", "train", 128, 1, 384, mask="none"),
    ]


def draw(rng):
    largest = _seconds(_case(None, "incoming", "infer", 128, 1, 2048))
    while True:
        op = rng.choice(("outgoing", "incoming", "outgoing", "incoming", "bidirectional", "transition"))
        mode = rng.choice(("infer", "infer", "train"))
        c = 64 if op != "transition" and rng.random() < 0.15 else 128
        b = rng.choice((1, 1, 1, 2, 4, 8))
        n = int(round(math.exp(rng.uniform(math.log(24), math.log(2048 if mode == "infer" else 1024)))))
        mask = "none" if op == "transition" else rng.choice(("none", "token", "token", "pair"))
        drop = mode == "train" and op != "transition" and c == 128 and rng.random() < 0.5
        if rng.random() < 0.5 or drop:
            n = max(24, (n + 7) // 8 * 8)  # crops are cut to round lengths, whole sequences are not
        case = _case(None, op, mode, c, b, n, mask, drop)
        if _seconds(case) <= largest:
            return case


def _hidden(case):
    """Contracted channels per direction."""
    return 64 if case["c"] == 64 and case["op"] == "bidirectional" else 128


def _shapes(case):
    c = case["c"]
    if case["op"] == "transition":
        return {"ln_in.weight": (c,), "ln_in.bias": (c,), "expand_a.weight": (4 * c, c), "expand_b.weight": (4 * c, c),
                "squeeze.weight": (c, 4 * c)}
    w = _hidden(case) * (2 if case["op"] == "bidirectional" else 1)
    return {"ln_pair.weight": (c,), "ln_pair.bias": (c,), "to_left.weight": (w, c), "to_left_gate.weight": (w, c),
            "to_right.weight": (w, c), "to_right_gate.weight": (w, c), "ln_out.weight": (w,), "ln_out.bias": (w,),
            "to_gate.weight": (c, c), "to_out.weight": (c, w)}


def _parameters(case, gen):
    """LayerNorm weights around one, small biases, linear weights of variance 1 / fan-in."""
    out = {}
    for key, shape in _shapes(case).items():
        r = torch.randn(*shape, generator=gen, device="cuda")
        if key.startswith("ln_"):
            out[key] = 1.0 + 0.1 * r if key.endswith("weight") else 0.02 * r
        else:
            out[key] = r * shape[1] ** -0.5
    return out


def _module(case):
    c, op = case["c"], case["op"]
    if op == "transition":
        return mw.Transition(c)
    if op == "bidirectional":
        return mw.BidirectionalTriangleMultiplication(c, _hidden(case))
    if case["mask"] == "pair":
        cls = mw.TriangleMultiplicationOutgoing if op == "outgoing" else mw.TriangleMultiplicationIncoming
        return cls(c, _hidden(case))
    return mw.TriangleMultiplication(c, _hidden(case), outgoing=op == "outgoing")


def _mask(case, gen):
    b, n = case["b"], case["n"]
    if case["mask"] == "none":
        return None
    if case["mask"] == "pair" and case["op"] != "bidirectional":
        return torch.rand(b, n, n, generator=gen, device="cuda") >= 0.1
    if b > 1:  # samples of different lengths, padded at the end
        length = torch.randint((5 * n + 7) // 8, n + 1, (b, 1), generator=gen, device="cuda")
        return torch.arange(n, device="cuda")[None, :] < length
    return torch.rand(b, n, generator=gen, device="cuda") >= 0.1


def _inputs(case, seed):
    """Parameters (fp32), pair tensor, mask, and for a training step the output's gradient and the dropout scale."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    b, n, c = case["b"], case["n"], case["c"]
    params = _parameters(case, gen)
    scale = 0.5 + 1.5 * torch.rand(c, generator=gen, device="cuda")
    z = torch.empty(b, n, n, c, device="cuda", dtype=torch.bfloat16)
    for i in range(b):  # (in slabs: the fp32 draw of a large pair tensor is never held whole)
        for r in range(0, n, 256):
            z[i, r : r + 256] = torch.randn(min(256, n - r), n, c, generator=gen, device="cuda") * scale
    mask, dy, drop_scale = _mask(case, gen), None, None
    if case["mode"] == "train":
        dy = torch.empty_like(z)
        for i in range(b):
            dy[i] = torch.randn(n, n, c, generator=gen, device="cuda") * 0.01
        if case["drop"]:
            keep = torch.rand(b, 1, n, c, generator=gen, device="cuda") >= 0.25
            drop_scale = keep.to(torch.bfloat16) / 0.75
    return params, z, mask, dy, drop_scale


def prepare(case, seed):
    params, z, mask, dy, drop_scale = _inputs(case, seed)
    state = {"z": z, "mask": mask}
    module = _module(case)
    module.load_state_dict(params)
    module = module.to("cuda")
    if case["mode"] == "infer":
        state["module"] = module.to(torch.bfloat16).eval()
        return state
    state["module"] = module.train()
    state["params"] = dict(module.named_parameters())
    z.requires_grad_(True)
    state["dy"] = dy
    if drop_scale is not None:
        state["drop_scale"] = drop_scale
    state["outgoing"] = {"outgoing": True, "incoming": False}.get(case["op"])
    return state


def run(state):
    z, mask, module = state["z"], state["mask"], state["module"]
    if "dy" not in state:
        with torch.no_grad():
            return module(z) if mask is None else module(z, mask)
    params = state["params"]
    if "drop_scale" in state:  # the functional entry point takes the dropout scale that a program drew
        pair = mask is not None and mask.dim() == 3
        y = trimul_train(z, params, None if pair else mask, outgoing=state["outgoing"], pair_mask=mask if pair else None,
                         drop_scale=state["drop_scale"])
    else:
        y = module(z) if mask is None else module(z, mask)
    grads = torch.autograd.grad(y, [z, *params.values()], state["dy"])
    return {"y": y.detach(), "z": grads[0], **dict(zip(params, grads[1:]))}


def _update64(case, p, z, valid, drop_scale):
    """The published operator on one sample ``z`` [N, N, C] in float64, residual included."""
    c = case["c"]
    if case["op"] == "transition":
        rows = []
        for zr in z.split(256):
            x = F.layer_norm(zr, (c,), p["ln_in.weight"], p["ln_in.bias"], 1e-5)
            h = F.silu(F.linear(x, p["expand_a.weight"])) * F.linear(x, p["expand_b.weight"])
            rows.append(zr + F.linear(h, p["squeeze.weight"]))
        return torch.cat(rows)
    x = F.layer_norm(z, (c,), p["ln_pair.weight"], p["ln_pair.bias"], 1e-5)
    left = torch.sigmoid(F.linear(x, p["to_left_gate.weight"])) * F.linear(x, p["to_left.weight"])
    right = torch.sigmoid(F.linear(x, p["to_right_gate.weight"])) * F.linear(x, p["to_right.weight"])
    if valid is not None:
        left, right = left * valid[..., None], right * valid[..., None]
    w = left.shape[-1]
    out = {"outgoing": w, "incoming": 0, "bidirectional": w // 2}[case["op"]]  # channels contracted over k of (i, k), (j, k)
    tri = []
    if out:
        tri.append(torch.einsum("ikd,jkd->ijd", left[..., :out], right[..., :out]))
    if out < w:
        tri.append(torch.einsum("kid,kjd->ijd", left[..., out:], right[..., out:]))
    del left, right
    t = F.layer_norm(torch.cat(tri, -1), (w,), p["ln_out.weight"], p["ln_out.bias"], 1e-5)
    del tri
    update = torch.sigmoid(F.linear(x, p["to_gate.weight"])) * F.linear(t, p["to_out.weight"])
    return z + (update if drop_scale is None else update * drop_scale)


def exact(case, seed):
    """What ``run`` returns, from the same inputs in float64 and one sample at a time (samples share the parameters only)."""
    params, z, mask, dy, drop_scale = _inputs(case, seed)
    train = case["mode"] == "train"
    p = {}
    for key, v in params.items():  # inference rounds the linear weights to bf16 once; the LayerNorms stay fp32
        p[key] = (v if train or key.startswith("ln_") else v.to(torch.bfloat16)).double().requires_grad_(train)
    out = {"y": torch.empty(z.shape, dtype=torch.float64, device="cuda")}
    if train:
        out["z"] = torch.empty_like(out["y"])
        out.update({key: torch.zeros_like(v) for key, v in p.items()})
    for i in range(case["b"]):
        valid = None
        if mask is not None:
            valid = mask[i] if mask.dim() == 3 else mask[i][:, None] & mask[i][None, :]
        drop = None if drop_scale is None else drop_scale[i].double()
        zi = z[i].double().requires_grad_(train)
        with torch.set_grad_enabled(train):
            y = _update64(case, p, zi, valid, drop)
            out["y"][i] = y.detach()
            if train:
                grads = torch.autograd.grad(y, [zi, *p.values()], dy[i].double())
                out["z"][i] = grads[0]
                for key, g in zip(p, grads[1:]):
                    out[key] += g
        del y
    return out if train else out["y"]


def work(case):
    """One read of every input and one write of every output; the multiply-adds of the published operator, and for a
    training step those of its two gradients (three times the forward: nothing that is recomputed counts)."""
    b, n, c = case["b"], case["n"], case["c"]
    cells = b * n * n
    weights = sum(math.prod(s) for s in _shapes(case).values())
    if case["op"] == "transition":
        flops = 2.0 * cells * 3 * 4 * c * c
    else:
        h, directions = _hidden(case), 2 if case["op"] == "bidirectional" else 1
        flops = 2.0 * cells * directions * n * h + 2.0 * cells * (5 * directions * h * c + c * c)
    masks = {"none": 0, "token": b * n, "pair": cells if case["op"] != "bidirectional" else b * n}[case["mask"]]
    if case["mode"] == "infer":
        return {"bytes": 2 * (2 * cells * c) + 2 * weights + masks, "flops": flops}
    drop = 2 * b * n * c if case["drop"] else 0
    return {"bytes": 4 * (2 * cells * c) + 8 * weights + masks + drop, "flops": 3.0 * flops}


def _seconds(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / 1.6e15)


def tolerance(case):
    """Against a float64 restatement of the operators (25 drawn shapes and six of the listed ones): outputs and gradients
    are within a relative 1.7e-3, which is the rounding of a bf16 result (2^-9 / sqrt(3) = 1.1e-3 and up, by how the values
    lie in their binades), largest difference 6.8e-3 of the value or of the root mean square; the fp32 parameter gradients
    are within 9e-4. Four times that."""
    return {"rel": 7e-3, "max": 2.8e-2}
