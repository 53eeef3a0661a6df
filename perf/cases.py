"""Training-step cases: what a program that trains with this framework runs, over the range of models, batches and options.

Every case is one step of the training loop through the public calls, as the trainer and the benchmark make them: the
random-walk batch of the step, forward + loss + backward, AdamW. The calls of a step are enqueued on the current stream and
nothing waits for them; a state keeps the step count, so successive passes are successive steps (other walks each time).
The puzzle is a set of random permutations and their inverses; the model has weights of ordinary scale, outputs that still
miss their labels, as early in a run, and AdamW moments that have run for a while. Everything comes from the seed.
"""
import math

import torch

import multigputrainmlp_b200 as mgt

LR = 1e-4

# precision: "fp16" / "bf16" operands on the tensor cores, "fp32_table" = fp16 linear layers with an fp32 table gradient
# (--input-grad-fp16 0), "fp32" = everything in fp32 (--linear-fp16 0 --input-grad-fp16 0, the default of the `mgt` CLI)
DEFAULTS = dict(state_len=72, values=72, outputs=1, k_max=29, precision="fp16", cross_entropy=False, batch_norm=False,
                mirror=True, weight_decay=0.0)


def _case(name, **kw):
    return dict(DEFAULTS, name=name, **kw)


def listed():
    return [
        # the trainer's own defaults: the smallest step there is, all launches and latency
        _case("smoke_64", hd1=8, hd2=8, blocks=1, batch=64, k_max=9),
        # the tiny residual model (plumbing runs, sweeps over seeds), in fp16 and in fp32
        _case("tiny_1024", hd1=256, hd2=64, blocks=2, batch=1024),
        _case("tiny_fp32_1024", hd1=256, hd2=64, blocks=2, batch=1024, precision="fp32"),
        # another puzzle: 54 positions of 6 colours (few classes per position), a mid-sized model
        _case("cube54_4096", state_len=54, values=6, hd1=1024, hd2=256, blocks=4, batch=4096),
        # sizes that are multiples of nothing, no fp16 mirror kept by the caller (--persistent-half-weights 0)
        _case("odd_no_mirror_5003", hd1=333, hd2=77, blocks=3, batch=5003, mirror=False),
        # depth classification with a ragged batch; a residual width that is a multiple of 8 only
        _case("classes_9001", hd1=1000, hd2=200, blocks=8, outputs=29, batch=9001, cross_entropy=True, weight_decay=0.01),
        # the p888 model on a small ragged batch (a strong-scaled rank, a fine-tuning run)
        _case("p888_3001", hd1=2560, hd2=224, blocks=16, batch=3001),
        # the headline configuration
        _case("p888_53248", hd1=2560, hd2=224, blocks=16, batch=53248),
        # ... with batch normalisation
        _case("p888_bn_53248", hd1=2560, hd2=224, blocks=16, batch=53248, batch_norm=True),
        # ... with the fp32 table gradient, and all in fp32
        _case("p888_fp32_table_16384", hd1=2560, hd2=224, blocks=16, batch=16384, precision="fp32_table"),
        _case("p888_fp32_8192", hd1=2560, hd2=224, blocks=16, batch=8192, precision="fp32"),
        # the wide and deep variant: bfloat16, cross-entropy on the depth, the largest hidden sizes
        _case("wide_bf16_131072", hd1=4096, hd2=512, blocks=32, outputs=29, batch=131072, precision="bf16", cross_entropy=True,
              weight_decay=0.01),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _layer_flops(c):
    """Multiply-adds x 2 of the dense layers, forward + both gradients, of one sample."""
    return 6.0 * (c["hd1"] * c["hd2"] + 2 * c["blocks"] * c["hd2"] ** 2 + c["hd2"] * c["outputs"])


def draw(rng):
    c = dict(DEFAULTS)
    c["precision"] = rng.choice(["fp16", "fp16", "fp16", "bf16", "fp32_table", "fp32"])
    if rng.random() < 0.4:  # another puzzle: permutations of all positions, or stickers of a few colours
        c["state_len"] = rng.randint(16, 72)
        c["values"] = c["state_len"] if rng.random() < 0.6 else rng.randint(4, 12)
    c["hd1"], c["hd2"], c["blocks"] = _log_int(rng, 64, 4096), _log_int(rng, 16, 512), rng.randint(1, 32)
    if rng.random() < 0.85:  # the trainer's padding of hidden sizes; the rest are sizes as they come
        c["hd1"], c["hd2"] = (c["hd1"] + 7) // 8 * 8, (c["hd2"] + 7) // 8 * 8
    c["k_max"] = rng.randint(5, 40)
    if rng.random() < 0.3:
        c["cross_entropy"] = c["precision"] in ("fp16", "bf16") and rng.random() < 0.7
        c["outputs"] = c["k_max"] if c["cross_entropy"] else rng.randint(2, 40)
    c["batch_norm"] = c["precision"] in ("fp16", "bf16") and rng.random() < 0.2
    c["mirror"] = rng.random() < 0.85
    c["weight_decay"] = rng.choice([0.0, 0.01])
    most = 1.0e11 if c["precision"] in ("fp32", "fp32_table") else 4.0e12
    c["batch"] = _log_int(rng, 64, max(64, min(131072, int(most / (_layer_flops(c) + 2.0 * c["state_len"] * c["values"] * c["hd1"])))))
    return c


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)

    def randn(n, std):
        return torch.randn(n, device=dev, generator=g) * std

    length, values, h1, h2, blocks, outputs, batch = (c[k] for k in ("state_len", "values", "hd1", "hd2", "blocks", "outputs", "batch"))
    shape = mgt.CudaMlpShape(length, values, h1, h2, blocks, outputs)
    rows = length * values
    parts = [randn(rows * h1, 0.8 / math.sqrt(length)), randn(h1, 0.05), randn(h1 * h2, math.sqrt(2.0 / h1)), randn(h2, 0.05)]
    for _ in range(blocks):  # residual branches smaller than the stream they add to
        parts += [randn(h2 * h2, math.sqrt(2.0 / h2)), randn(h2, 0.05), randn(h2 * h2, 0.25 / math.sqrt(h2 * blocks)), randn(h2, 0.02)]
    parts += [randn(h2 * outputs, 1.0 / math.sqrt(h2)), randn(outputs, 1.0 if c["cross_entropy"] else 0.1)]
    if c["batch_norm"]:
        for layer in range(blocks + 1):  # branches whose scale has grown little from zero, the usual start
            parts += [(0.05 if layer else 1.0) * (1.0 + randn(h2, 0.1)), randn(h2, 0.1) + (0.05 if layer else 1.0)]
    w = torch.cat(parts)
    total = w.numel()
    moves = torch.zeros(18, 80, dtype=torch.uint8, device=dev)
    for i in range(0, 18, 2):
        perm = torch.randperm(length, device=dev, generator=g)
        moves[i, :length] = perm.to(torch.uint8)
        moves[i + 1, :length] = torch.argsort(perm).to(torch.uint8)
    target = torch.zeros(80, dtype=torch.uint8, device=dev)
    target[:length] = (torch.arange(length, device=dev) * values // length).to(torch.uint8)
    fp32 = c["precision"] == "fp32"
    half_table = c["precision"] not in ("fp32", "fp32_table")
    engine = mgt.Engine(torch.cuda.current_device())
    if engine.set_train_options(bf16=c["precision"] == "bf16", cross_entropy=c["cross_entropy"], batch_norm=c["batch_norm"]) != 0:
        raise RuntimeError("train options")
    running = None
    if c["batch_norm"]:
        running = torch.zeros(blocks + 1, 2, h2, device=dev)
        running[:, 1] = 1.0
        engine.set_batch_norm_state(running, 0.1, 1)
    floats = mgt.mlp_loss_grad_workspace_floats(shape, batch, 1, half_table, not fp32, batch_norm=c["batch_norm"])
    depth = torch.zeros(batch, device=dev)
    return {
        "shape": shape, "batch": batch, "outputs": outputs, "total": total, "engine": engine, "seed": seed, "step": 100,
        "walk": mgt.RandomWalkKernelConfig(batch, 1, c["k_max"], 18, length, 80), "weight_decay": c["weight_decay"],
        "half_table": half_table, "half_linear": not fp32, "w": w, "w_half": w.half() if c["mirror"] and not fp32 else None,
        "m": randn(total, 1e-4), "v": 1e-6 * (0.5 + torch.rand(total, device=dev, generator=g)), "grad": torch.zeros(total, device=dev),
        "loss": torch.zeros(1, device=dev), "moves": moves, "target": target,
        "states": torch.zeros(batch, 80, dtype=torch.uint8, device=dev), "depth": depth,
        "labels": depth if outputs == 1 else torch.zeros(batch * outputs, device=dev),
        "meta": torch.zeros(batch, 16, dtype=torch.uint8, device=dev), "running": running,
        "workspace": torch.empty(floats, device=dev), "floats": floats,
    }


def run(s):
    """One training step: walk batch -> loss and gradients -> AdamW."""
    step = s["step"]
    s["step"] = step + 1
    status = mgt.launch_random_walk_kernel(s["walk"], s["seed"], 0, step, 0, s["moves"], s["target"], s["states"], s["depth"], s["meta"])
    if s["outputs"] > 1:
        status |= mgt.launch_expand_scalar_labels(s["depth"], s["batch"], s["outputs"], s["labels"])
    status |= s["engine"].launch_mlp_loss_grad(s["shape"], s["w"], s["w_half"], s["states"], s["labels"], s["batch"], s["loss"], s["grad"],
                                               s["workspace"], s["floats"], use_half_input_grad=s["half_table"],
                                               use_half_linear=s["half_linear"])
    adamw = mgt.AdamWKernelConfig(s["total"], step + 1, LR, weight_decay=s["weight_decay"])
    if s["w_half"] is not None:
        status |= mgt.launch_adamw_kernel_with_half_mirror(adamw, s["w"], s["w_half"], s["grad"], s["m"], s["v"])
    else:
        status |= mgt.launch_adamw_kernel(adamw, s["w"], s["grad"], s["m"], s["v"])
    if status != 0:
        raise RuntimeError("a call of the step failed")
    out = {k: s[k] for k in ("loss", "grad", "w", "m", "v", "states", "depth", "meta")}
    for k in ("w_half", "running"):
        if s[k] is not None:
            out[k] = s[k]
    return out


def work(case):
    """The arithmetic of the model (the embedding as the sparse sums it is, forward and gradient); the parameters, gradient
    and moments once through memory, and the walk batch."""
    c = dict(DEFAULTS, **case)
    h2, batch = c["hd2"], c["batch"]
    params = c["state_len"] * c["values"] * c["hd1"] + c["hd1"] + c["hd1"] * h2 + h2 + 2 * c["blocks"] * (h2 * h2 + h2) + h2 * c["outputs"] + c["outputs"]
    if c["batch_norm"]:
        params += 2 * (c["blocks"] + 1) * h2
    mirror = 2 if c["mirror"] and c["precision"] != "fp32" else 0
    return {"bytes": params * (7 * 4 + mirror) + batch * (80 + 4 + 16), "flops": batch * (_layer_flops(c) + 2.0 * c["state_len"] * c["hd1"])}


def tolerance(case):
    """Walks, depths and generator states are whole numbers and stay the same. The gradients pass through two roundings to the
    operand format per layer (11 bits in fp16, 8 in bfloat16), and a rounding that falls the other way can open or close a
    ReLU; in fp32 only the order of the sums differs."""
    c = dict(DEFAULTS, **case)
    if c["precision"] == "fp32":
        return {"rel": 5e-5, "max": 2e-2}
    return {"rel": 1.5e-2, "max": 0.7} if c["precision"] == "bf16" else {"rel": 5e-3, "max": 0.5}
