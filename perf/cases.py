"""The work that programs built on this framework have it do on one GPU, as cases that can be timed.

Every case is a pass of one kind of program through the framework's public entry points:

* ``train``    - ``Trainer.train_step``: token ids in pinned host memory in, loss out (what ``bench.py`` and the training
                 entry points do every step).  Forward, backward, the in-place gradients and the fused AdamW.
* ``reduce``   - ``LocalCluster.allreduce_``: a compressed (or cast) mean all-reduce of one gradient bucket, all ranks of
                 the collective on this GPU.  It is the kernel that the DDP hooks launch once per bucket and rank.
* ``records``  - the ``dynamiQ_mee_{b}bit_dynamic_bitrate`` chain on the same buckets: centre the superchunks, sum their
                 statistics, choose widths, plan, one mixed-width collective, add the means back, move the controller.
* ``codec``    - ``RhtCodec``: encode a bucket, add a local one at a hop, decode (the standalone codec operators).
* ``thc``      - one partition of the THC baseline as one rank computes it: whole-vector rotation, quantise, dequantise,
                 rotation back.
* ``eden``     - EDEN compress and decompress.

Sizes are those of the repository's configurations: the model registry and ``bench.py``'s batch shapes, gradient
tensors of 1 MB to 256 MB (the all-reduce sweep), 25 MB DDP buckets, THC partitions of at most 2^23 elements.
"""
from __future__ import annotations

import math

import torch

from dynamiq_sigcomm_artifact_b200 import bitalloc, ops
from dynamiq_sigcomm_artifact_b200.ops.fwht import fwht_pow2
from dynamiq_sigcomm_artifact_b200.parallel.baselines import THC_T
from dynamiq_sigcomm_artifact_b200.parallel.eden import Eden
from dynamiq_sigcomm_artifact_b200.parallel.fused import LocalCluster, RhtCodec
from dynamiq_sigcomm_artifact_b200.train.engine import TrainConfig, Trainer

SMS = 148
THREADS = 512  # block size of the operator benchmark (train/bench_allreduce.py)

# registry name -> (layers, hidden, query heads, kv heads, inner, matrices of the MLP, vocabulary, longest sequence, task)
MODELS = {
    "gpt2-tiny": (2, 128, 4, 4, 512, 2, 1024, 128, "causal"),
    "llama-tiny": (2, 128, 4, 2, 256, 3, 1024, 128, "causal"),
    "bert-tiny": (2, 128, 4, 4, 256, 2, 1024, 128, "mlm"),
    "gpt2-small": (12, 768, 12, 12, 3072, 2, 50257, 1024, "causal"),
    "bert-base": (12, 768, 12, 12, 3072, 2, 30522, 512, "mlm"),
    "llama-1.2b": (16, 2048, 32, 8, 8192, 3, 128256, 2048, "causal"),
}


def listed():
    return [
        # the smallest training step (tests, smoke runs, hyper-parameter sweeps of toy models): host and launch latency
        {"name": "train-gpt2-tiny", "kind": "train", "model": "gpt2-tiny", "batch": 2, "seq": 128},
        # the headline configuration: GPT-2 small, micro-batch 8, context 1024
        {"name": "train-gpt2-small", "kind": "train", "model": "gpt2-small", "batch": 8, "seq": 1024},
        # masked LM: BERT-base, batch 16, sequence 512, masking on the device
        {"name": "train-bert-base", "kind": "train", "model": "bert-base", "batch": 16, "seq": 512},
        # the large configuration: Llama-style 1.2 B, micro-batch 4, sequence 2048
        {"name": "train-llama-1.2b", "kind": "train", "model": "llama-1.2b", "batch": 4, "seq": 2048},
        # one 1 MB bucket, two ranks: the latency end of the all-reduce sweep
        {"name": "reduce-1mb-5bit", "kind": "reduce", "n": 262_144, "world": 2, "codec": "rht", "bits": 5,
         "topology": "direct", "dtype": "fp32"},
        # 64 MB per rank, the default method (dynamiQ_aee_5bit, direct topology), four ranks
        {"name": "reduce-64mb-5bit", "kind": "reduce", "n": 1 << 24, "world": 4, "codec": "rht", "bits": 5,
         "topology": "direct", "dtype": "fp32"},
        # a ragged bf16 bucket of a DDP user over eight ranks, 8-bit butterfly
        {"name": "reduce-ragged-8bit-bf16", "kind": "reduce", "n": 3_000_001, "world": 8, "codec": "rht", "bits": 8,
         "topology": "butterfly", "dtype": "bf16"},
        # the uncompressed bf16 hook on a 25 MB bucket over the ring
        {"name": "reduce-25mb-bf16-wire", "kind": "reduce", "n": 6_553_600, "world": 4, "codec": "cast", "bits": 16,
         "topology": "ring", "dtype": "fp32"},
        # the reference's record format: mean-centred superchunks with 8 / 4 / 2-bit codes, controlled average width
        {"name": "records-25mb-mee-5bit", "kind": "records", "n": 6_553_600, "world": 4, "bits": 5, "topology": "direct"},
        # standalone codec operators on a 64 MB gradient
        {"name": "codec-64mb-5bit", "kind": "codec", "n": 1 << 24, "bits": 5},
        # one THC partition of a 12 MB gradient (padded to 2^22 values)
        {"name": "thc-3m", "kind": "thc", "n": 3_000_001, "levels": 31},
        # EDEN on a ragged gradient of a few MB
        {"name": "eden-2m-4bit", "kind": "eden", "n": 2_000_003, "bits": 4},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "reduce", "reduce", "reduce", "records", "codec", "thc", "eden"])
    if kind == "train":
        model = rng.choice(sorted(MODELS))
        longest = MODELS[model][7]
        batch = _spread(rng, 1, {"llama-1.2b": 4, "bert-base": 16}.get(model, 8))
        return {"kind": kind, "model": model, "batch": batch, "seq": _spread(rng, 24, longest)}
    if kind == "reduce":
        codec, widths = rng.choice([("rht", (4, 5, 8)), ("rht", (4, 5, 8)), ("cast", (16, 32)), ("mx", (4, 6, 8))])
        return {"kind": kind, "n": _spread(rng, 200_000, 1 << 24), "world": rng.choice([2, 4, 8]), "codec": codec,
                "bits": rng.choice(widths), "topology": rng.choice(["ring", "butterfly", "direct"]),
                "dtype": rng.choice(["fp32", "fp32", "bf16"])}
    if kind == "records":
        return {"kind": kind, "n": _spread(rng, 200_000, 1 << 24), "world": rng.choice([2, 4]), "bits": rng.choice([4, 5, 6]),
                "topology": rng.choice(["butterfly", "direct"])}
    if kind == "codec":
        return {"kind": kind, "n": _spread(rng, 200_000, 1 << 26), "bits": rng.choice([3, 4, 5, 6, 8])}
    if kind == "thc":
        return {"kind": kind, "n": _spread(rng, 3_000, 1 << 23), "levels": rng.choice([15, 31])}
    return {"kind": kind, "n": _spread(rng, 100_000, 1 << 24), "bits": rng.randint(1, 8)}


def _gradient(n, seed, dtype=torch.float32):
    """N(0, 1) with a lognormal scale (sigma 2) per 1024 values: gradients of layers of very different size."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, device="cuda", generator=g)
    scale = torch.exp(2.0 * torch.randn((n + 1023) // 1024, device="cuda", generator=g))
    return (x * scale.repeat_interleave(1024)[:n]).to(dtype)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        with torch.device("cuda"):  # weights are initialised where they will live
            trainer = Trainer(TrainConfig(model=case["model"], method="dynamiQ_aee_5bit", micro_batch=case["batch"],
                                          seq_len=case["seq"], task=MODELS[case["model"]][8], seed=seed))
        batch = torch.randint(0, MODELS[case["model"]][6], (case["batch"], case["seq"]), dtype=torch.int64,
                              generator=torch.Generator().manual_seed(seed)).pin_memory()
        params = [p for p in trainer.model.parameters() if p.dim() == 2]
        blocks = max(p.numel() for p in params[1:])
        # the tied embedding and the largest matrices of the blocks (run() returns at most 64 tensors)
        watched = [params[0]] + [p for p in params[1:] if p.numel() == blocks]
        return {"trainer": trainer, "batch": batch, "watched": [p.detach() for p in watched]}
    n = case["n"]
    if kind == "reduce":
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        world = case["world"]
        return {"cluster": LocalCluster(world, n, ctas=SMS // world, threads=THREADS), "step": 0, "seed": seed,
                "grads": [_gradient(n, 64 * seed + r, dtype) for r in range(world)],
                "how": (case["bits"], case["topology"], case["codec"])}
    if kind == "records":
        world = case["world"]
        ops.require()
        padded = (n + 255) // 256 * 256  # centred superchunks are whole
        return {"cluster": LocalCluster(world, padded, ctas=SMS // world, threads=THREADS), "step": 0, "seed": seed,
                "grads": [_gradient(n, 64 * seed + r) for r in range(world)], "topology": case["topology"],
                "controller": bitalloc.DeviceBitrateController(case["bits"], "cuda")}
    if kind == "codec":
        return {"codec": RhtCodec(case["bits"], n, seed=seed, ctas=SMS, threads=THREADS), "step": 0,
                "x": _gradient(n, 2 * seed), "local": _gradient(n, 2 * seed + 1)}
    if kind == "thc":
        d = 1 << (n - 1).bit_length()
        x = torch.zeros(d, device="cuda")
        x[:n] = _gradient(n, seed)
        # largest norm of the ranks, and the coordinate that is sent exactly
        return {"x": x, "stats": torch.stack([x.norm(), x.sum() / math.sqrt(d)]), "levels": case["levels"], "step": 0,
                "seed": seed}
    if kind == "eden":
        return {"eden": Eden(case["bits"], seed=seed), "x": _gradient(n, seed), "step": 0}
    raise ValueError(kind)


def run(state):
    if "trainer" in state:
        trainer = state["trainer"]
        loss = trainer.train_step(state["batch"])
        return {"loss": loss, "gradients": trainer.reducer.arena, "weights": state["watched"]}
    if "controller" in state:
        return _records(state)
    if "cluster" in state:
        bits, topology, codec = state["how"]
        state["step"] += 1
        return state["cluster"].allreduce_(state["grads"], bits, topology, seed=state["seed"], step=state["step"],
                                           codec=None if codec == "rht" else codec)
    if "codec" in state:
        codec, step = state["codec"], state["step"]
        state["step"] += 1
        sent = codec.compress(state["x"], step=step)
        hop = codec.dec_comp(sent, state["local"], step=step)
        return {"sent": sent, "hop": hop, "sum": codec.decompress(hop, state["x"].numel(), step=step)}
    if "eden" in state:
        eden, step = state["eden"], state["step"]
        state["step"] += 1
        words, scale, n = eden.compress(state["x"], step=step)
        return {"words": words, "scale": scale, "x": eden.decompress((words, scale, n), step=step)}
    dq, x, stats = ops.require(), state["x"], state["stats"]
    scale = THC_T / math.sqrt(x.numel())
    state["step"] += 1
    y = fwht_pow2(x, normalize=True)
    dq.thc_quantize_(y, stats, 1, scale, state["levels"], 0, state["step"], state["seed"])
    dq.thc_dequantize_(y, stats, 1, scale, state["levels"])
    return {"rotated": y, "back": fwht_pow2(y, normalize=True)}


def _records(state):
    """One bucket of ``dynamiQ_mee_{b}bit_dynamic_bitrate`` on every rank, as parallel/superchunk.py runs it."""
    dq, cluster, grads, controller = ops.require(), state["cluster"], state["grads"], state["controller"]
    world, seed = len(grads), state["seed"]
    state["step"] += 1
    step = state["step"]
    centred = [dq.superchunk_center(g, world) for g in grads]
    stats = [s for _, s in centred]
    cluster.allreduce_([s.view(-1) for s in stats], 32, "direct", seed=seed, step=step, bucket_id=2, codec="cast",
                       post_scale=1.0)
    widths = controller.widths(stats[0])
    plan = dq.superchunk_plan(widths)
    cluster.allreduce_([r for r, _ in centred], 8, state["topology"], seed=seed, step=step, bucket_id=3,
                       codec="scmix_mee", plan=plan)
    for g, (r, s) in zip(grads, centred):
        dq.superchunk_add_mean(r, s[:, 0].contiguous(), g)
    controller.end_of_step()
    return {"grads": grads, "widths": widths, "controller": controller.state}


def work(case):
    kind = case["kind"]
    if kind == "train":
        layers, hidden, heads, kv, inner, mats, vocab, _, task = MODELS[case["model"]]
        head_dim = hidden // heads
        block = hidden * (heads + 2 * kv) * head_dim + hidden * hidden + mats * hidden * inner
        matmul = layers * block + vocab * hidden + (hidden * hidden if task == "mlm" else 0)
        tokens = case["batch"] * case["seq"]
        attention = 4 * layers * tokens * case["seq"] * hidden * (1.0 if task == "mlm" else 0.5)
        # weights and both moments read and written, gradients written; the activations could stay on the chip
        return {"bytes": 28.0 * matmul, "flops": 3.0 * (2.0 * matmul * tokens + attention)}
    n = case["n"]
    if kind == "reduce":
        return {"bytes": 2.0 * n * case["world"] * (2 if case["dtype"] == "bf16" else 4), "flops": 0.0}
    if kind == "records":
        return {"bytes": 8.0 * n * case["world"], "flops": 0.0}
    if kind == "codec":  # x, local and the sum; two messages written, each read once
        return {"bytes": 12.0 * n + 4.0 * n * case["bits"] / 8, "flops": 0.0}
    if kind == "thc":  # x read, the two returned vectors written, the first of them read once
        return {"bytes": 16.0 * (1 << (n - 1).bit_length()), "flops": 0.0}
    return {"bytes": 8.0 * n + 2.0 * n * case["bits"] / 8, "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "train":  # bf16 activations and bf16 gradients of activations through every layer
        return {"rel": 2e-2}
    if kind == "reduce" and case["dtype"] == "bf16":
        return {"rel": 4e-3}  # one rounding to bf16
    if kind == "thc":  # a coordinate on the boundary of two bins may fall on either side
        return {"rel": 1e-3, "max": 0.9}
    if kind == "eden":  # the same
        return {"rel": 1e-3, "max": 0.5, "differ": 1e-4}
    return {"rel": 1e-5}  # seeded stochastic codes: the same bytes, fp32 sums
