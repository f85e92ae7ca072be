"""ProtX distillation student: the encoder without the MLM head, followed by an optional
projection to the teacher width and a T5-style (RMS) norm
(reference: src/nanoplm/distillation/models/student/model.py:50-109). Parameter names follow the
reference / HF ModernBertModel (`embeddings.*`, `layers.N.*`, `final_norm`, `proj`, `proj_norm`)."""
from __future__ import annotations

from pathlib import Path
from typing import Optional

import numpy as np
import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.nn.modules.module import _has_any_global_hook

from nanoplm_b200.config.schema import StudentConfig
from nanoplm_b200.data.tokenizer import StudentTokenizer
from nanoplm_b200.models.encoder import (Attention, BatchContext, EncoderModel, Linear, Norm, _own_forward,
                                         position_ids_from_cu_seqlens)
from nanoplm_b200.ops import functional as ops
from nanoplm_b200.ops import kernels as K


# Tokens and bytes of activations up to which embed_sequences joins batches. Longer runs gain nothing more (GEMMs of 32 768 rows
# fill 256 tiles of 128 rows a column of tiles).
_EMBED_TOKENS, _EMBED_BYTES = 32768, 512 << 20


class ProtX(EncoderModel):
    def __init__(self, cfg: StudentConfig, tokenizer: Optional[StudentTokenizer] = None):
        self.tokenizer = tokenizer or StudentTokenizer()
        self.student_config = cfg
        mc = cfg.to_model_config(self.tokenizer.vocab_size)
        super().__init__(mc)
        self.proj = self.proj_norm = None
        if cfg.projection_layer:
            self.proj = Linear(cfg.hidden_size, cfg.teacher_dim, False)
            self.proj_norm = Norm(cfg.teacher_dim, 1e-6, rms=True)
        self.init_weights()

    @torch.no_grad()
    def init_weights(self) -> None:
        import math
        cfg = self.config
        bound = math.sqrt(3.0 / cfg.hidden_size)
        nn.init.normal_(self.embeddings.tok_embeddings.weight, 0.0, 0.02)
        for layer in self.layers:
            nn.init.uniform_(layer.attn.Wqkv.weight, -bound, bound)
            nn.init.uniform_(layer.attn.Wo.weight, -bound / 4, bound / 4)
            nn.init.uniform_(layer.mlp.Wi.weight, -bound, bound)
            nn.init.uniform_(layer.mlp.Wo.weight, -bound / 4, bound / 4)
        if self.proj is not None:
            nn.init.uniform_(self.proj.weight, -bound, bound)

    def forward(self, input_ids, attention_mask=None, training_mode: bool = False, cu_seqlens=None,
                position_ids=None):
        """Padded (B, S) or flat ids. Returns {"last_hidden_state"} in the input's layout; with
        training_mode the projected + normed states (teacher width)."""
        x, pad_info = self._states(input_ids, attention_mask, training_mode, cu_seqlens, position_ids)
        if pad_info is not None:
            indices, B, S = pad_info
            full = torch.zeros((B * S, x.shape[-1]), dtype=x.dtype, device=x.device)
            full = full.index_copy(0, indices, x)
            x = full.view(B, S, -1)
        return {"last_hidden_state": x}

    def _states(self, input_ids, attention_mask, training_mode, cu_seqlens=None, position_ids=None):
        """(states of the real tokens [T, width], (their indices, B, S) of a padded batch or None)."""
        pad_info = None
        if input_ids.dim() == 2:
            B, S = input_ids.shape
            if attention_mask is None:
                attention_mask = torch.ones_like(input_ids)
            if position_ids is None and ops.unpad_takes(input_ids, attention_mask):
                ids, indices, position_ids, cu_seqlens = ops.unpad(input_ids, attention_mask)
            else:
                keep = attention_mask.reshape(-1).bool()
                indices = torch.nonzero(keep, as_tuple=False).flatten()
                ids = input_ids.reshape(-1)[indices]
                lens = attention_mask.sum(dim=-1, dtype=torch.int32)
                cu_seqlens = F.pad(torch.cumsum(lens, 0, dtype=torch.int32), (1, 0))
            pad_info = (indices, B, S)
        else:
            ids = input_ids
        T = ids.shape[0]
        if position_ids is None:
            position_ids = position_ids_from_cu_seqlens(cu_seqlens, T, ids.device)
        ctx = BatchContext(cu_seqlens.to(ids.device), position_ids.to(ids.device), T)
        x, _ = EncoderModel.forward(self, ids, ctx)
        if training_mode and self.proj is not None:
            x = self.proj_norm(self.proj(x))
        return x, pad_info

    def packed_states(self, input_ids, attention_mask):
        """(states in the training mode [T, width], int64 indices of their rows among the B * S positions) of a padded batch
        on a GPU, for callers that need no padded output; None where somebody observes calls of this module."""
        if not (type(self).forward is _FORWARD and "forward" not in self.__dict__ and not self._forward_hooks
                and not self._forward_pre_hooks and not self._backward_hooks and not self._backward_pre_hooks
                and not _has_any_global_hook() and self.final_norm.weight.dtype == torch.bfloat16
                and input_ids.dim() == 2 and ops.unpad_takes(input_ids, attention_mask)):
            return None
        x, (indices, _, _) = self._states(input_ids, attention_mask, True)
        return x, indices

    # ---- utilities of the reference student (model.py:111-497) ---------------------------------
    def num_parameters(self) -> int:
        return sum(p.numel() for p in self.parameters())

    def parameter_breakdown(self) -> dict:
        groups = {"embeddings": 0, "attention": 0, "mlp": 0, "norms": 0, "projection": 0, "other": 0}
        for name, p in self.named_parameters():
            if name.startswith("embeddings.tok"):
                groups["embeddings"] += p.numel()
            elif ".attn." in name:
                groups["attention"] += p.numel()
            elif ".mlp." in name:
                groups["mlp"] += p.numel()
            elif "norm" in name:
                groups["norms"] += p.numel()
            elif name.startswith("proj"):
                groups["projection"] += p.numel()
            else:
                groups["other"] += p.numel()
        groups["total"] = sum(groups.values())
        return groups

    def _embeds_packed(self, device: torch.device) -> bool:
        """Whether embed_sequences may hand the model flat ids: bf16 on a GPU, and nothing that observes the padded
        call (a forward of a subclass, of this instance or put on the class, hooks on this module or on all modules)."""
        w = self.final_norm.weight
        return (device.type == "cuda" and w.dtype == torch.bfloat16 and w.shape[0] % 8 == 0
                and type(self).forward is _FORWARD and "forward" not in self.__dict__
                and not self._forward_hooks and not self._forward_pre_hooks and not _has_any_global_hook())

    def _join_tokens(self) -> int:
        """Tokens up to which embed_sequences may run several batches as one (0: not at all). Between them lies padding whose rows
        have no keys: the attention kernel for 64-wide heads gives such rows zeros, the dense form that other widths take
        gives NaN, which the next layer would spread, and needs scores of the square of the tokens. Experts see how many tokens
        a call has."""
        cfg = self.config
        for l in self.layers:       # (a dozen layers before the first launch: no look-ups through Module.__getattr__)
            a = l._modules.get("attn")
            if not _own_forward(l) or l.is_moe or type(a) is not Attention or a.head_dim != 64:
                return 0
            qkv = a._modules["Wqkv"]
            w = qkv._parameters.get("weight")
            if type(qkv) is not Linear or w is None or w.dtype != torch.bfloat16:
                return 0
        # two copies of the streams and a layer's tensors beside them: 13.3 KB at 512 channels, 26.6 at 1024, 19.5 for four streams of
        # 512, where the allocator's peak is 8.2, 16.5 and 16.5 a token
        per_token = 2 * (cfg.hidden_size * (7 + 2 * cfg.mhc_streams) + 2 * cfg.intermediate_size)
        return min(_EMBED_TOKENS, _EMBED_BYTES // per_token)

    def _pack_batches(self, batches: list[list[str]]) -> tuple[np.ndarray, np.ndarray, list[bool]]:
        """(ids, lengths, which of the sequences are real) of several batches one after the other. Every batch starts on a
        multiple of 256 tokens, behind padding: the attention's tiles then cut a batch where they cut it alone, and the
        padding has no keys, as rows past the end have none, so that a batch's results have the bits they have alone."""
        if len(batches) == 1:
            return *self.tokenizer.pack(batches[0]), [True] * len(batches[0])
        ids, lens, real = [], [], []
        for i, b in enumerate(batches):
            tokens, n = self.tokenizer.pack(b)
            ids.append(tokens)
            lens.append(n)
            real += [True] * len(n)
            pad = -len(tokens) % 256 if i + 1 < len(batches) else 0
            if pad:
                ids.append(np.full(pad, self.tokenizer.pad_token_id, np.int32))
                lens.append(np.array([pad], np.int32))
                real.append(False)
        return np.concatenate(ids), np.concatenate(lens), real

    def _embed_packed(self, ids: np.ndarray, lens: np.ndarray, device, real: list[bool]):
        """(hidden states [T, C] of the tokens, device cu_seqlens) of a packed host batch: ids, positions, the tokens' key
        ranges and offsets go over in one copy from pinned memory and nothing waits for the device."""
        T, B = len(ids), len(lens)
        Tp = (T + 3) // 4 * 4                                  # every part starts on 16 bytes
        host = torch.empty(4 * Tp + B + 1, dtype=torch.int32, pin_memory=True)
        buf = host.numpy()
        cu = np.zeros(B + 1, np.int32)
        np.cumsum(lens, out=cu[1:])
        at = np.arange(T, dtype=np.int32)
        start, end = np.repeat(cu[:-1], lens), np.repeat(cu[1:], lens)
        if not all(real):
            pad = ~np.repeat(np.array(real), lens)
            start[pad] = end[pad] = at[pad]
        buf[:T] = ids
        buf[Tp:Tp + T] = at - start
        buf[2 * Tp:2 * Tp + T] = start
        buf[3 * Tp:3 * Tp + T] = end
        buf[4 * Tp:] = cu
        dev = host.to(device, non_blocking=True)
        cu_dev = dev[4 * Tp:]
        ctx = BatchContext(cu_dev, dev[Tp:Tp + T], T, bounds=(dev[2 * Tp:2 * Tp + T], dev[3 * Tp:3 * Tp + T]))
        h, _ = EncoderModel.forward(self, dev[:T], ctx)
        return h, cu_dev

    def _embed_run(self, ids: np.ndarray, lens: np.ndarray, real: list[bool], per_token: bool, device):
        """(device rows, how many of them each real sequence has; -1 for the mean of a stretch of padding) of a packed host
        batch."""
        h, cu = self._embed_packed(ids, lens, device, real)
        if not per_token:
            return K.segment_mean(h, cu, drop_last=1), [1 if r else -1 for r in real]
        ends, lens = np.cumsum(lens).tolist(), lens.tolist()    # the residues' rows, without the trailing </s> of every sequence
        keep = torch.cat([torch.arange(e - n, e - 1) for n, e, r in zip(lens, ends, real) if r])
        return h[keep.to(device)], [n - 1 for n, r in zip(lens, real) if r]

    @torch.no_grad()
    def embed_sequences(self, sequences: list[str], batch_size: int = 16, per_token: bool = False,
                        device: Optional[torch.device] = None) -> list[torch.Tensor]:
        """Mean-pooled (EOS excluded) or per-token embeddings for raw sequences.

        batch_size is the number of sequences that are padded to a common length where padding is needed, and what
        bounds the memory there. A bf16 model with 64-wide heads on a GPU takes packed sequences: whole batches run together
        up to 32 768 tokens and 512 MiB of activations, with the results that they have one by one, and one by one where
        the memory for that is not there."""
        device = device or next(self.parameters()).device
        # (walking all modules to set a flag that is set already costs more than several layers' launches, and so does
        # looking at it through `modules()`, which remembers whom it has met)
        was_training, watched, walk = False, False, [self]
        while walk:
            m = walk.pop()
            was_training |= m.training
            watched |= bool(m._forward_hooks) or bool(m._forward_pre_hooks) or "forward" in m.__dict__
            walk += [c for c in m._modules.values() if c is not None]
        restore = self.training
        if was_training:
            self.eval()
        packed = self._embeds_packed(torch.device(device))
        out, waiting, rows = [], [], 0

        def collect():
            """One copy to the host for all results that wait on the device; every sequence gets its own tensor."""
            nonlocal rows
            if waiting:
                host = (waiting[0][0] if len(waiting) == 1 else torch.cat([t for t, _ in waiting])).cpu()
                lens = [n for _, ns in waiting for n in ns]
                for n, part in zip(lens, host.split([abs(n) for n in lens])):
                    if n >= 0:                                  # (negative: the mean of a stretch of padding)
                        out.append(part.float() if per_token else part[0].clone())
                waiting.clear()
                rows = 0

        direct = packed and type(self.tokenizer) is StudentTokenizer and self.tokenizer.packs()
        plain = lambda b: type(b) is list and all(type(t) is str for t in b)
        most = 0 if watched else None       # tokens of joined batches; a hook on some part may count them
        i, end = 0, len(sequences) if range(0, 1, batch_size) else 0       # (a step of 0 is an error, a negative one no steps)
        while i < end:
            first, batch, flat, joined = i, sequences[i:i + batch_size], None, []
            i += batch_size
            if direct and plain(batch):
                # Packed rows neither know their batch nor pad it: further batches join while they fit, and a layer's launches
                # fill the chip. 91 proteins of 46 000 tokens at 512 channels took 36 layers of 8 000 rows, one to two
                # waves of tiles a GEMM.
                joined = [batch]
                tokens = sum(map(len, batch)) + len(batch)
                while i < end:
                    if most is None:
                        most = self._join_tokens()
                    more = sequences[i:i + batch_size]
                    tokens += 255 + sum(map(len, more)) + len(more) if most and plain(more) else most + 1
                    if tokens > most:
                        break
                    joined.append(more)
                    i += batch_size
                flat = self._pack_batches(joined)
            else:
                enc = self.tokenizer(batch, padding=True, return_tensors="pt")
                ids, mask = enc["input_ids"], enc["attention_mask"]
                # the real tokens first, at least one, then padding
                if (packed and not ids.is_cuda and bool(mask[:, 0].all())
                        and bool((mask[:, :-1] >= mask[:, 1:]).all())):
                    flat = ids.numpy()[mask.numpy().astype(bool)], mask.sum(dim=1).numpy(), [True] * len(mask)
            if flat is not None:
                try:
                    waiting.append(self._embed_run(*flat, per_token, device))
                except torch.OutOfMemoryError:
                    if len(joined) < 2:
                        raise
                    i, most = first, 0          # what fits one by one still runs
                    continue
                rows += waiting[-1][0].shape[0]
                if rows >= 65536:   # bounds what waits on the device
                    collect()
                continue
            collect()
            ids, mask = ids.to(device), mask.to(device)
            h = self(ids, mask)["last_hidden_state"].float()
            for b in range(ids.shape[0]):
                n = int(mask[b].sum()) - 1          # drop the trailing </s>
                out.append(h[b, :n].cpu() if per_token else h[b, :n].mean(0).cpu())
        collect()
        if was_training:
            self.train(restore)
        return out


_FORWARD = ProtX.forward


def inspect_checkpoint_architecture(path: str | Path) -> dict:
    """Infers the student architecture from a saved state dict (safetensors or torch)."""
    p = Path(path)
    if p.suffix == ".safetensors":
        from safetensors.torch import load_file
        sd = load_file(str(p))
    else:
        sd = torch.load(p, map_location="cpu", weights_only=True)
    layers = sorted({int(k.split(".")[1]) for k in sd if k.startswith("layers.")})
    hidden = sd["embeddings.tok_embeddings.weight"].shape[1]
    info = {"hidden_size": hidden, "vocab_size": sd["embeddings.tok_embeddings.weight"].shape[0],
            "num_hidden_layers": len(layers), "projection_layer": "proj.weight" in sd,
            "num_parameters": sum(v.numel() for v in sd.values())}
    if layers:
        info["intermediate_size"] = sd[f"layers.{layers[0]}.mlp.Wo.weight"].shape[1]
    return info


def calculate_model_parameters(model: torch.nn.Module) -> dict:
    """Total and trainable parameter counts (reference: student/model.py, parameter utilities)."""
    total = sum(p.numel() for p in model.parameters())
    trainable = sum(p.numel() for p in model.parameters() if p.requires_grad)
    return {"total": total, "trainable": trainable, "frozen": total - trainable}


def print_parameter_breakdown(model: "ProtX") -> dict:
    """Logs the per-group parameter counts of a student and returns them."""
    from nanoplm_b200.utils.logging import logger
    groups = model.parameter_breakdown()
    total = max(1, groups["total"])
    for name, n in groups.items():
        if name != "total":
            logger.info(f"{name:>12s}: {n:>12,d}  ({100.0 * n / total:5.1f} %)")
    logger.info(f"{'total':>12s}: {groups['total']:>12,d}")
    return groups


def load_and_generate_embeddings(checkpoint: str | Path, sequences: list[str], cfg: Optional[StudentConfig] = None,
                                 batch_size: int = 16, per_token: bool = False,
                                 device: Optional[torch.device] = None) -> list[torch.Tensor]:
    """Loads a saved student (safetensors or torch state dict) and embeds raw sequences: mean-pooled
    over the residues (the trailing </s> excluded) or one vector per residue
    (reference: student/model.py:111-248). Without `cfg` the architecture is inferred from the file;
    the head count defaults to hidden_size / 64."""
    p = Path(checkpoint)
    if p.is_dir():
        p = p / ("model.safetensors" if (p / "model.safetensors").exists() else "pytorch_model.bin")
    if p.suffix == ".safetensors":
        from safetensors.torch import load_file
        sd = load_file(str(p))
    else:
        sd = torch.load(p, map_location="cpu", weights_only=True)
    if cfg is None:
        info = inspect_checkpoint_architecture(p)
        cfg = StudentConfig(hidden_size=info["hidden_size"], intermediate_size=info.get("intermediate_size", 2 * info["hidden_size"]),
                            num_hidden_layers=info["num_hidden_layers"],
                            num_attention_heads=max(1, info["hidden_size"] // 64),
                            projection_layer=info["projection_layer"])
    model = ProtX(cfg)
    missing, unexpected = model.load_state_dict(sd, strict=False)
    if unexpected:
        raise KeyError(f"unexpected keys in student checkpoint: {sorted(unexpected)[:5]}")
    device = device or torch.device("cuda" if torch.cuda.is_available() else "cpu")
    model = model.to(device)
    if device.type == "cuda":
        model = model.to(torch.bfloat16)
    return model.embed_sequences(sequences, batch_size=batch_size, per_token=per_token, device=device)
