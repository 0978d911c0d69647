"""The work this package is used for, as cases that can be timed: decode steps, prefill and scoring (forward
without gradients), training steps (forward and backward), and the Vision-Mamba2 forward pass.

A case is a dict of plain values.  ``kind`` says how the package is called:

  "forward"  ``mamba2_ssd_fwd`` without gradients
  "train"    ``mamba2_ssd_fwd`` with gradients, then ``torch.autograd.grad`` for every differentiable input
  "vision"   ``VisionMamba2`` (12 blocks, width 192), inference

``features`` of an SSD case: "basic" (softplus only) or "full" (D skip connection, z gate, dt_bias and dt limits as
well); ``start`` adds an initial state, ``final`` asks for the final state, ``policy`` is what autograd keeps.
Inputs follow the benchmark configurations: x, B, C ~ N(0,1), dt ~ U[0,1), A = -U[0,1), fp32 throughout.
"""
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "mamba-ascendc_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

import ascend_kernel as ak  # noqa: E402
from ascend_kernel.vmamba2 import VisionMamba2, VisionMamba2Config  # noqa: E402


def _ssd(name, kind, shape, features="basic", start=False, final=True, policy="save"):
    b, l, h, p, n, chunk, g = shape
    case = dict(kind=kind, batch=b, seqlen=l, heads=h, headdim=p, dstate=n, chunk=chunk, groups=g, features=features,
                start=start, final=final, policy=policy)
    return dict(name=name, **case) if name else case


def listed():
    return [
        # one generation step: one token of each of 16 sequences, the state goes in and comes out
        _ssd("decode_one_token", "forward", (16, 1, 24, 64, 128, 128, 1), "full", start=True),
        # benchmark configuration 0: the shortest forward that fills a tile; launches and host work count
        _ssd("forward_one_tile", "forward", (1, 128, 2, 64, 128, 128, 1)),
        # benchmark configuration 1: the same for a training step
        _ssd("train_one_tile", "train", (1, 128, 2, 64, 64, 64, 1)),
        # benchmark configuration 2: scoring a batch, no final state
        _ssd("forward_batch_n128", "forward", (4, 2048, 16, 64, 128, 128, 4), final=False),
        # prefill of one long prompt by a layer whose heads share one group, as most models of this kind have it
        _ssd("prefill_one_group", "forward", (1, 8192, 32, 64, 64, 64, 1), "full"),
        # the SSD of a Vision-Mamba2 block in training: 4 images, six heads, one group
        _ssd("train_vision_block", "train", (4, 4096, 6, 64, 64, 64, 1), "full", final=False),
        # training with state size 128
        _ssd("train_n128", "train", (4, 2048, 16, 64, 128, 128, 4)),
        # training with a ragged length and headdim 32
        _ssd("train_ragged_p32", "train", (4, 2000, 32, 32, 64, 64, 4)),
        # training with every optional input, activations recomputed in backward
        _ssd("train_full_recompute", "train", (2, 4096, 64, 64, 64, 64, 16), "full", start=True, policy="recompute"),
        # one rank's share of the H256 training step on eight GPUs
        _ssd("train_h32_share", "train", (8, 4096, 32, 64, 64, 64, 8)),
        # benchmark configuration 3: the whole H256 training step on one GPU
        _ssd("train_h256", "train", (8, 4096, 256, 64, 64, 64, 64)),
        # benchmark configuration 4: one GPU's images of the batch
        dict(name="vision_forward", kind="vision", batch=4, image=1024),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    family = rng.choice(["decode", "forward", "forward", "train", "train", "train", "vision"])
    if family == "vision":
        return dict(kind="vision", batch=rng.randint(1, 4), image=16 * rng.randint(14, 64))
    groups = rng.choice([1, 1, 2, 4, 8])
    heads = groups * _log_int(rng, max(1, 4 // groups), 32 // groups) if groups < 8 else 8 * _log_int(rng, 1, 16)
    p = rng.choice([64, 64, 64, 32, 128])
    n = rng.choice([64, 64, 128, 32])
    features = rng.choice(["basic", "full"])
    if family == "decode":
        return _ssd(None, "forward", (_log_int(rng, 1, 64), rng.choice([1, 1, 1, 2, 5, 8]), heads, p, n, 64, groups),
                    features, start=True)
    batch = _log_int(rng, 1, 8)
    length = _log_int(rng, 100, 16384)
    if rng.random() < 0.6:
        length = max(128, length // 128 * 128)
    while batch * length * heads * max(p, 64) * max(n, 64) > 8 * 4096 * 64 * 64 * 64:
        length = max(128, length // 256 * 128)
        batch = max(1, batch // 2) if length == 128 else batch
    return _ssd(None, family, (batch, length, heads, p, n, rng.choice([64, 128]), groups), features,
                start=rng.random() < 0.3, final=rng.random() < 0.6,
                policy=rng.choice(["save", "save", "recompute"]) if family == "train" else "save")


_LIMITS = (1e-3, 1.0)  # dt limits of the full feature set


def prepare(case, seed):
    if case["kind"] == "vision":
        devices = [torch.cuda.current_device()]
        with torch.random.fork_rng(devices=devices), torch.device("cuda"):
            torch.manual_seed(seed)
            net = VisionMamba2(VisionMamba2Config(image_size=case["image"])).eval()
            return {"case": case, "net": net, "images": torch.randn(case["batch"], 3, case["image"], case["image"])}
    gen = torch.Generator(device="cuda").manual_seed(seed)
    b, l, h, p, n, g = (case[k] for k in ("batch", "seqlen", "heads", "headdim", "dstate", "groups"))

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device="cuda")

    tensors = {"x": normal(b, l, h, p), "dt": uniform(b, l, h), "A": -uniform(h), "B": normal(b, l, g, n),
               "C": normal(b, l, g, n)}
    if case["features"] == "full":
        tensors["D"] = normal(h)
        tensors["z"] = normal(b, l, h, p)
        tensors["dt_bias"] = 0.1 * normal(h)
    if case["start"]:
        tensors["initial_states"] = normal(b, h, p, n)
    state = {"case": case, "tensors": tensors}
    if case["kind"] == "train":
        for t in tensors.values():
            t.requires_grad_(True)
        state["upstream"] = [normal(b, l, h, p)] + ([normal(b, h, p, n)] if case["final"] else [])
    return state


def _ssd_call(case, t):
    full = case["features"] == "full"
    return ak.mamba2_ssd_fwd(t["x"], t["dt"], t["A"], t["B"], t["C"], case["chunk"], D=t.get("D"), z=t.get("z"),
                             dt_bias=t.get("dt_bias"), dt_softplus=True, dt_limit=_LIMITS if full else (0.0, float("inf")),
                             initial_states=t.get("initial_states"), return_final_state=case["final"])


def run(state):
    case = state["case"]
    if case["kind"] == "vision":
        with torch.no_grad():
            return state["net"](state["images"])
    if case["kind"] == "forward":
        with torch.no_grad():
            return _ssd_call(case, state["tensors"])
    previous = ak.set_save_policy(case["policy"])
    try:
        got = _ssd_call(case, state["tensors"])
        outputs = list(got) if case["final"] else [got]
        grads = torch.autograd.grad(outputs, list(state["tensors"].values()), state["upstream"])
    finally:
        ak.set_save_policy(previous)
    return [o.detach() for o in outputs] + list(grads)


def work(case):
    """Each tensor of the call once (a training step reads its inputs once in each direction), and the products of
    the chunked algorithm at the case's own chunk length; backward is twice the forward."""
    if case["kind"] == "vision":
        c = VisionMamba2Config(image_size=case["image"])
        b, l = case["batch"], c.tokens
        proj = c.d_model * (2 * c.d_inner + 2 * c.ngroups * c.d_state + c.nheads) + c.d_inner * c.d_model
        conv = c.d_conv * (c.d_inner + 2 * c.ngroups * c.d_state)
        ssd = _flops(b, l, c.nheads, c.headdim, c.d_state, c.chunk_size, c.ngroups)
        embed = 3 * c.patch * c.patch * c.d_model
        weights = c.depth * (proj + conv) + embed + c.d_model * c.num_classes
        return {"bytes": 4.0 * (b * 3 * case["image"] ** 2 + weights + b * c.num_classes),
                "flops": c.depth * (2.0 * b * l * (proj + conv) + ssd) + 2.0 * b * l * embed}
    b, l, h, p, n, g = (case[k] for k in ("batch", "seqlen", "heads", "headdim", "dstate", "groups"))
    full = case["features"] == "full"
    x, state = b * l * h * p, b * h * p * n
    inputs = x * (2 if full else 1) + b * l * h + 2 * b * l * g * n + h * (3 if full else 1) + (state if case["start"] else 0)
    outputs = x + (state if case["final"] else 0)
    flops = _flops(b, l, h, p, n, case["chunk"], g)
    if case["kind"] == "train":
        return {"bytes": 4.0 * (inputs + outputs + inputs + outputs + inputs), "flops": 3.0 * flops}
    return {"bytes": 4.0 * (inputs + outputs), "flops": flops}


def _flops(b, l, h, p, n, chunk, g):
    t = min(chunk, l)
    return float(b) * l * (g * 2 * t * n + h * (2 * t * p + 4 * n * p))


def tolerance(case):
    """Against the same path in 64 bits.  Operands carry 16 mantissa bits (bf16 hi + lo) and sums are fp32: 6.3e-6 on
    every output of a forward call.  In a training step the gradients of A and dt_bias are sums of tens of thousands
    of terms of either sign, and their relative error is that of the terms divided by what is left of the sum:
    2e-5 to 3.4e-4 seen with the seeds tried.  The network's patch embedding is the framework's convolution, which
    uses TF32 by default: 1.3e-4 on the logits.  Stated: four times these."""
    return {"rel": {"forward": 2.5e-5, "train": 1.4e-3, "vision": 5e-4}[case["kind"]]}
