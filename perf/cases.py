"""What the performance of this framework is measured on: training steps, evaluation and embedding
calls through the public entry points, from a single protein to the full micro-batch.

A case is a dict of plain values. `kind` picks the entry point:

  embed    ProtX.embed_sequences: raw sequences in, one pooled vector per protein out (host to host)
  logits   ProtEncoderMLM.forward on a padded batch without labels (inference, evaluation)
  train    TrainStep.step_from_host: pinned host micro-batches in, loss out; forward, backward, optimizer
  distill  one optimizer step of the distillation student against given teacher embeddings
  teacher  T5EncoderTeacher.forward, the frozen teacher of on-the-fly distillation

Weights are random, but the output projections that a fresh model starts at zero are given values,
as they have after the first few hundred steps. Sequences are drawn at natural amino-acid
frequencies with uniform lengths, as the package's synthetic data is.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nanoplm_b200.config.schema import (ModelConfig, MoEConfig, PretrainingConfig, StudentConfig, TeacherConfig)
from nanoplm_b200.data.collators import PackingCollator
from nanoplm_b200.data.packing import pack_ffd
from nanoplm_b200.data.synthetic import synthetic_sequences, synthetic_token_sequences
from nanoplm_b200.data.tokenizer import ProtTokenizer
from nanoplm_b200.models.encoder import ProtEncoderMLM
from nanoplm_b200.models.student import ProtX
from nanoplm_b200.models.teacher import T5EncoderTeacher
from nanoplm_b200.ops import functional as ops
from nanoplm_b200.parallel.engine import AdamWHyper, ShardedEngine
from nanoplm_b200.parallel.muon import MuonEngine
from nanoplm_b200.runtime.distill import DistillDataCollator, distillation_loss
from nanoplm_b200.runtime.pretrain import TrainStep
from nanoplm_b200.runtime.schedule import WarmupLinearSchedule

DEV = torch.device("cuda:0")
MLM_PROB = 0.15


# ------------------------------------------------------------------------------------------ cases
def _train(name, hidden, inter, layers, seqs, lo, hi, variant="default", optimizer="adamw", accum=1):
    c = {"kind": "train", "hidden": hidden, "inter": inter, "layers": layers, "seqs": seqs, "lo": lo, "hi": hi,
         "variant": variant, "optimizer": optimizer, "accum": accum}
    return dict(c, name=name) if name else c


def _student(kind, name, hidden, inter, layers, seqs, lo, hi, variant="default", batch=16):
    c = {"kind": kind, "hidden": hidden, "inter": inter, "layers": layers, "seqs": seqs, "lo": lo, "hi": hi,
         "variant": variant, "batch": batch}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one protein through the default distilled student: the interactive call, all latency
        _student("embed", "embed_one", 512, 1024, 6, 1, 230, 240),
        # a small FASTA file embedded with the default student and the default batch size, lengths ragged
        _student("embed", "embed_many", 512, 1024, 6, 91, 20, 1000),
        # scoring a padded batch of long and short proteins with the default encoder (logits of every position)
        {"name": "logits_padded", "kind": "logits", "hidden": 1024, "inter": 2048, "layers": 16, "seqs": 9,
         "lo": 20, "hi": 1000},
        # a small encoder on a few short proteins, two micro-batches a step: where launches and host work count
        _train("train_small", 256, 512, 3, 23, 20, 200, accum=2),
        # the default encoder with the template's 32 sequences per micro-batch
        _train("train_default_32", 1024, 2048, 16, 32, 20, 512),
        # the default encoder on the full micro-batch of the throughput configuration (128 rows of 512)
        _train("train_default_208", 1024, 2048, 16, 208, 20, 512),
        # the same encoder with e4m3 linear layers (`pretraining.fp8: true`)
        _train("train_fp8_208", 1024, 2048, 16, 208, 20, 512, variant="fp8"),
        # mixture of experts: every second MLP 64 experts, top-2; long sequences up to 1024
        _train("train_moe_100", 1024, 2048, 8, 100, 20, 1000, variant="moe"),
        # the Muon optimizer on the default encoder, a small global batch
        _train("train_muon_16", 1024, 2048, 16, 16, 20, 512, optimizer="muon"),
        # default distillation recipe: 512 x 6 student, 64 sequences padded to 512
        _student("distill", "distill_default_64", 512, 1024, 6, 64, 20, 511),
        # convolution + hyper-connection student (768 x 12) on the same batch
        _student("distill", "distill_conv_mhc_64", 768, 1536, 12, 64, 20, 511, variant="conv_mhc"),
        # the 24-layer T5-style teacher on a distillation batch, padding removed from host-known lengths
        {"name": "teacher_64", "kind": "teacher", "layers": 24, "seqs": 64, "lo": 20, "hi": 511},
    ]


#: most sequences a drawn case may have at 512 tokens each, per kind of work (keeps it below the listed ones)
_DRAW_TOP = {"default": 160, "fp8": 128, "moe": 96, "conv_mhc": 48, "rmsnorm": 160}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["embed", "logits", "train", "train", "train", "distill", "teacher"])
    hi = rng.choice([rng.randint(60, 260), rng.randint(261, 511), rng.randint(512, 1000)])
    lo = rng.choice([20, 20, rng.randint(21, hi - 20)])
    if kind == "embed":
        hidden, inter, layers = rng.choice([(512, 1024, 6), (512, 1024, 6), (768, 1536, 12), (256, 512, 4)])
        return _student(kind, None, hidden, inter, layers, _log_int(rng, 1, 160), lo, hi,
                        batch=rng.choice([8, 16, 16, 32, 64]))
    if kind == "logits":
        hidden, inter, layers = rng.choice([(1024, 2048, 16), (768, 1536, 12), (512, 1024, 8)])
        return {"kind": kind, "hidden": hidden, "inter": inter, "layers": layers, "seqs": _log_int(rng, 1, 48),
                "lo": lo, "hi": hi}
    if kind == "teacher":
        return {"kind": kind, "layers": 24, "seqs": max(1, int(_log_int(rng, 1, 60) * 511 / max(hi, 511))),
                "lo": lo, "hi": hi}
    if kind == "distill":
        variant = rng.choice(["default", "conv_mhc"])
        hidden, inter, layers = rng.choice([(512, 1024, 6), (768, 1536, 12), (384, 768, 8)])
        hi = min(hi, 511)
        return _student(kind, None, hidden, inter, layers, _log_int(rng, 4, 60), min(lo, hi - 20), hi, variant)
    variant = rng.choice(["default", "default", "rmsnorm", "fp8", "moe", "conv_mhc"])
    hidden, inter, layers = rng.choice([(1024, 2048, 16), (1024, 2048, 16), (768, 1536, 12), (512, 1024, 8),
                                        (256, 512, 4)])
    if variant == "moe":
        hidden, inter, layers = rng.choice([(1024, 2048, 8), (512, 1024, 6)])
    top = max(8, int(_DRAW_TOP[variant] * 512 / max(hi, 512)))
    seqs = _log_int(rng, 4, top)
    if variant == "moe":            # enough tokens for 64 experts
        hi, seqs = max(hi, 400), max(seqs, 60)
        lo = min(lo, hi - 20)
    optimizer = rng.choice(["adamw", "adamw", "adamw", "muon", "normuon"]) if variant in ("default", "rmsnorm") else "adamw"
    return _train(None, hidden, inter, layers, seqs, lo, hi, variant, optimizer, rng.choice([1, 1, 2]))


# ---------------------------------------------------------------------------------------- prepare
def _fill_output_projections(model, std=0.02):
    """Projections that start at zero (every block would be the identity) get values."""
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith(("attn.Wo.weight", "mlp.Wo.weight", "experts_Wo")):
                p.normal_(0.0, std)


def _model_config(case):
    extra = {}
    if case.get("variant") == "moe":
        extra["moe"] = MoEConfig(num_experts=64, top_k=2, expert_intermediate_size=512, every_n_layers=2)
    elif case.get("variant") == "conv_mhc":
        extra.update(conv_kernel_size=7, mhc_streams=4)
    elif case.get("variant") == "rmsnorm":
        extra["norm_type"] = "rmsnorm"
    return ModelConfig(hidden_size=case["hidden"], intermediate_size=case["inter"], num_hidden_layers=case["layers"],
                       num_attention_heads=case["hidden"] // 64, vocab_size=32, max_position_embeddings=1024, **extra)


def _student_model(case):
    kw = dict(conv_kernel_size=7, mhc_streams=4) if case["variant"] == "conv_mhc" else {}
    return ProtX(StudentConfig(hidden_size=case["hidden"], intermediate_size=case["inter"],
                               num_hidden_layers=case["layers"], num_attention_heads=case["hidden"] // 64, **kw))


def _lengths_seed(seed):
    return int(seed) % (2 ** 31)


def _prepare_train(case, seed):
    tok = ProtTokenizer()
    with torch.device(DEV):
        model = ProtEncoderMLM(_model_config(case), tok)
    _fill_output_projections(model)
    hyper = AdamWHyper(lr=1e-3, max_grad_norm=1.0)
    if case["optimizer"] == "adamw":
        engine = ShardedEngine(model, hyper, DEV, compute_dtype=torch.bfloat16)
    else:
        engine = MuonEngine(model, hyper, PretrainingConfig(dataset_dir="x", optimizer=case["optimizer"]), DEV)
    model.train()
    sched = WarmupLinearSchedule(1e-3, 10_000, 1_000_000)
    sched.load_state_dict({"last_epoch": 100})           # early in the warm-up: the rate is 1e-5 and rises
    width = case["hi"] + 1
    batches = []
    for a in range(case["accum"]):
        s = _lengths_seed(seed * 7 + a)
        seqs = synthetic_token_sequences(case["seqs"], case["lo"], case["hi"], seed=s)
        lens = np.asarray([len(x) for x in seqs], np.int32)
        # the static layout holds every sequence and ends in a padding tail of about a sixth, as in production
        rows = max(int(pack_ffd(lens, width)[3]), int(math.ceil(1.18 * lens.sum() / width)))
        coll = PackingCollator(tok, width, MLM_PROB, target_rows=rows, batch_size=len(seqs), seed=s)
        b = coll([{"input_ids": torch.from_numpy(x)} for x in seqs])
        b.pop("labels")                                   # masked_idx / masked_labels carry the same information
        batches.append({k: (v.pin_memory() if torch.is_tensor(v) else v) for k, v in b.items()})
    return {"step": TrainStep(model, engine, sched, DEV), "engine": engine, "batches": batches,
            "fp8": case["variant"] == "fp8"}


def _prepare_distill(case, seed):
    with torch.device(DEV):
        student = _student_model(case)
    engine = ShardedEngine(student, AdamWHyper(lr=1e-3, weight_decay=0.01), DEV, decay_all=True)
    student.train()
    width = 512
    coll = DistillDataCollator(True, width)
    b = coll([{"raw_sequence": s} for s in synthetic_sequences(case["seqs"], case["lo"], case["hi"],
                                                               seed=_lengths_seed(seed))])
    batch = {k: b[k].to(DEV) for k in ("input_ids", "attention_mask")}
    # what the teacher just left on the device: unit-scale embeddings, zeros at the padding
    emb = torch.randn((case["seqs"], width, 1024), device=DEV)
    batch["teacher_embeddings"] = (emb * batch["attention_mask"][:, :, None]).to(torch.bfloat16)
    return {"student": student, "engine": engine, "batch": batch}


def prepare(case, seed):
    torch.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "train":
        st = _prepare_train(case, int(seed))
    elif kind == "distill":
        st = _prepare_distill(case, int(seed))
    elif kind == "embed":
        with torch.device(DEV):
            model = _student_model(case)
        st = {"model": model.to(torch.bfloat16).eval(), "batch": case["batch"],
              "seqs": synthetic_sequences(case["seqs"], case["lo"], case["hi"], seed=_lengths_seed(seed))}
    elif kind == "logits":
        tok = ProtTokenizer()
        with torch.device(DEV):
            model = ProtEncoderMLM(_model_config(case), tok)
        _fill_output_projections(model)
        enc = tok(synthetic_sequences(case["seqs"], case["lo"], case["hi"], seed=_lengths_seed(seed)),
                  padding="max_length", max_length=case["hi"] + 1, return_tensors="pt")
        st = {"model": model.to(torch.bfloat16).eval(), "ids": enc["input_ids"].to(DEV),
              "mask": enc["attention_mask"].to(DEV)}
    else:
        with torch.device(DEV):
            model = T5EncoderTeacher(TeacherConfig(num_layers=case["layers"]), random_init=False)
        with torch.no_grad():
            for name, p in model.named_parameters():
                if p.ndim >= 2:      # T5 folds the attention scale into q
                    p.normal_(0.0, p.shape[-1] ** -0.5 * (128 ** -0.5 if name.endswith("SelfAttention.q.weight") else 1.0))
        coll = DistillDataCollator(True, case["hi"] + 1)
        b = coll([{"raw_sequence": s} for s in synthetic_sequences(case["seqs"], case["lo"], case["hi"],
                                                                   seed=_lengths_seed(seed))])
        st = {"model": model.to(torch.bfloat16), "ids": b["teacher_input_ids"].to(DEV),
              "mask": b["teacher_attention_mask"].to(DEV), "lengths": b["teacher_lengths"]}
    st["kind"] = kind
    return st


# -------------------------------------------------------------------------------------------- run
def _updated(engine):
    """Weights and first moments (the gradients, as the optimizer has taken them in). The flat moments come
    in runs of tensors with gradients of like size: the embeddings, every layer, the vectors, the last norm.
    With experts the layers are one run: an expert that a tie sends one token more sees few tokens in all."""
    experts = any("experts" in s.name for s in engine.slots)
    runs, last = [], None
    for s in engine.slots:
        layer = s.name.split("layers.")[1].split(".")[0] if "layers." in s.name and s.decay and not experts else ""
        group = (s.decay, layer, "embeddings" in s.name, "proj_norm" in s.name)
        if group != last:
            runs.append(s.offset)
            last = group
    runs.append(engine.total)
    return {"weights": engine.master, "momentum": [engine.exp_avg[a:b] for a, b in zip(runs, runs[1:])]}


def run(state):
    kind = state["kind"]
    ops.set_fp8(state.get("fp8", False))
    if kind == "train":
        loss = state["step"].step_from_host(state["batches"])
        return {"loss": loss, **_updated(state["engine"])}
    if kind == "distill":
        loss = distillation_loss(state["student"], state["batch"])
        loss.backward()
        norm = state["engine"].step(1e-5, 1)
        return {"loss": loss.detach(), "grad_norm": norm, **_updated(state["engine"])}
    if kind == "embed":
        return torch.stack(state["model"].embed_sequences(state["seqs"], batch_size=state["batch"]))
    if kind == "logits":
        with torch.no_grad():
            return state["model"](state["ids"], state["mask"])["logits"]
    return state["model"](state["ids"], state["mask"], lengths=state["lengths"])


# ------------------------------------------------------------------------------------------- work
def _tokens(case):
    """Expected tokens and sum of squared lengths of a batch (lengths uniform, one special token)."""
    lo, hi = case["lo"] + 1, case["hi"] + 1
    mean = (lo + hi) / 2
    return case["seqs"] * mean, case["seqs"] * (mean * mean + (hi - lo) ** 2 / 12)


def _encoder_forward(hidden, inter, layers, T, T2, variant):
    """(multiply-add FLOPs, weights) of the encoder blocks; a third of the layers attend globally, the
    others to at most 129 neighbours."""
    glob = (layers + 2) // 3
    local = min(T2, 129 * T)
    flops = layers * T * 8 * hidden * hidden + 4 * hidden * (glob * T2 + (layers - glob) * local)
    weights = layers * 4 * hidden * hidden
    dense = layers
    if variant == "moe":
        dense = layers - layers // 2
        flops += (layers // 2) * T * (2 * 6 * hidden * 512 + 2 * hidden * 64)
        weights += (layers // 2) * (64 * 3 * hidden * 512 + 64 * hidden)
    flops += dense * T * 6 * hidden * inter
    weights += dense * 3 * hidden * inter
    if variant == "conv_mhc":       # 4 streams, two sites a layer: read, write and 4 x 4 mixing
        flops += layers * T * hidden * (2 * 7 + 2 * (2 * 4 + 2 * 4 + 2 * 16 + 2 * 24))
        weights += layers * hidden * (7 + 2 * 25)
    return flops, weights


def work(case):
    kind = case["kind"]
    T, T2 = _tokens(case)
    if kind == "teacher":
        d, ff, inner = 1024, 16384, 32 * 128
        flops = case["layers"] * (T * (8 * d * inner + 4 * d * ff) + 4 * inner * T2)
        weights = case["layers"] * (4 * d * inner + 2 * d * ff)
        return {"bytes": 2 * weights + 8 * T + 2 * d * case["seqs"] * (case["hi"] + 1), "flops": flops}
    h = case["hidden"]
    flops, weights = _encoder_forward(h, case["inter"], case["layers"], T, T2, case.get("variant", "default"))
    if kind == "embed":
        batches = -(-case["seqs"] // case["batch"])
        return {"bytes": batches * 2 * weights + 8 * T + 4 * case["seqs"] * h, "flops": flops}
    if kind == "logits":
        return {"bytes": 2 * weights + 8 * T + 64 * case["seqs"] * case["hi"], "flops": flops + T * (2 * h * h + 64 * h)}
    steps = case.get("accum", 1)
    if kind == "distill":
        flops += 2 * T * h * 1024
        extra = case["seqs"] * 512 * 1024 * 2
        weights += h * 1024
    else:
        flops += MLM_PROB * T * (2 * h * h + 64 * h)
        extra = 8 * T
        weights += h * h
    flops *= 3 * steps
    if case.get("optimizer") in ("muon", "normuon"):
        for r, c in ((3 * h, h), (h, h), (2 * case["inter"], h), (h, case["inter"])):
            m, n = min(r, c), max(r, c)
            flops += case["layers"] * 5 * (4 * m * m * n + 2 * m ** 3)
    # weights and optimizer state are read and written once a step: fp32 master, two moments, bf16 copy
    return {"bytes": weights * (2 * steps + 24 + 2) + steps * extra, "flops": flops}


def tolerance(case):
    """bf16 activations and fp32 sums, compared with the same path on other kernels (other tiles, other orders
    of summation, another attention kernel): about four times the relative difference seen there, in the worst
    output. Losses and weights agree far better than the moments, which are gradients."""
    kind, variant = case["kind"], case.get("variant")
    if kind == "embed":
        return {"rel": 0.01, "max": 0.08}            # seen 0.0024 / 0.017
    if kind in ("logits", "distill") or variant in ("fp8", "moe", "conv_mhc"):
        return {"rel": 0.03, "max": 1.0 - 1e-6}      # seen 0.006 (moe, ties in the routing) to 0.021 (e4m3) / 0.9
    return {"rel": 0.02, "max": 0.8}                 # seen 0.008 / 0.31; teacher against its restatement 0.010 / 0.07
