"""The framework's everyday work, as cases for timing: training steps, evaluation, serving and the lookup on its own.

Every case goes through the entry points a program uses (tasks and partitioners, the predictor, the embedding module,
the sequence layers).  Geometries are those of the experiments under `recml_b200/examples` and of the benchmarks; item
and id tables are cut to at most two million rows so that several states fit one GPU.  Inputs have the distributions of
`recml_b200.data.synthetic` (Zipf ids, log-normal dense features, power-law lengths, exponential time gaps) and are
drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from recml_b200 import embedding as emb
from recml_b200 import serving
from recml_b200.data import synthetic
from recml_b200.examples import dlrm_experiment, hstu_experiment, sasrec_experiment
from recml_b200.layers import hstu as hstu_layers
from recml_b200.layers import mamba as mamba_layers
from recml_b200.models import dlrm as dlrm_model
from recml_b200.training import optim_factory, partitioning

DEVICE = "cuda"
CRITEO_VOCAB = synthetic.CRITEO_VOCAB_SIZES
CRITEO_BAGS = synthetic.CRITEO_MULTI_HOT_SIZES


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed() -> list[dict]:
  return [
      # the headline training step: one GPU takes the whole global batch
      {"name": "dlrm_train_65536", "kind": "dlrm_train", "batch": 65536, "rows": 2_000_000},
      # one GPU's share of that batch on an eight-GPU node
      {"name": "dlrm_train_8192", "kind": "dlrm_train", "batch": 8192, "rows": 2_000_000},
      # the batch of the stand-alone DLRM trainer (not a multiple of a tile)
      {"name": "dlrm_train_4224", "kind": "dlrm_train", "batch": 4224, "rows": 1_000_000},
      # the small configuration: eight one-id features, full-rank cross layers, dense Adagrad
      {"name": "dlrm_tiny_256", "kind": "dlrm_tiny", "batch": 256, "tables": 8, "rows": 1000, "dim": 16},
      # serving: host batch in, logits out
      {"name": "dlrm_predict_500", "kind": "dlrm_predict", "batch": 500, "rows": 1_000_000},
      # the lookup and its row update alone: jagged mean-pooled bags
      {"name": "embedding_16384x64", "kind": "embedding", "batch": 16384, "tables": 8, "rows": 1_000_000, "dim": 64,
       "bag": 12, "combiner": "mean", "optimizer": "rowwise_adagrad"},
      # generative retrieval: 128 sequences of power-law length, mean about 512
      {"name": "hstu_train_128x512", "kind": "hstu_train", "sequences": 128, "mean_len": 512, "max_len": 4096,
       "heads": 4, "layers": 8, "rows": 2_000_000, "negatives": 512},
      # its small configuration
      {"name": "hstu_train_8x40", "kind": "hstu_train", "sequences": 8, "mean_len": 40, "max_len": 256,
       "heads": 1, "layers": 2, "rows": 2000, "negatives": 32},
      # forward only: user states from a batch of histories
      {"name": "hstu_encode_40x300", "kind": "hstu_encode", "sequences": 40, "mean_len": 300, "max_len": 2048,
       "heads": 4, "layers": 4},
      # causal transformer recommender
      {"name": "sasrec_train_512x200", "kind": "sasrec_train", "batch": 512, "length": 200, "rows": 2_000_000},
      # rank of the held-out item among the whole vocabulary
      {"name": "sasrec_eval_512", "kind": "sasrec_eval", "batch": 512, "length": 200, "rows": 1_000_000},
      # state-space recommender blocks, forward and backward
      {"name": "mamba_train_256x200", "kind": "mamba_train", "batch": 256, "length": 200, "layers": 2},
  ]


def _log_int(rng, lo: int, hi: int) -> int:
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
  kind = rng.choice(["dlrm_train", "dlrm_tiny", "dlrm_predict", "embedding", "hstu_train", "hstu_encode",
                     "sasrec_train", "sasrec_eval", "mamba_train"])
  if kind == "dlrm_train":
    return {"kind": kind, "batch": _log_int(rng, 512, 60000), "rows": _log_int(rng, 100_000, 2_000_000)}
  if kind == "dlrm_tiny":
    return {"kind": kind, "batch": _log_int(rng, 64, 4096), "tables": rng.randint(4, 12),
            "rows": _log_int(rng, 100, 5000), "dim": rng.choice([16, 32, 64])}
  if kind == "dlrm_predict":
    return {"kind": kind, "batch": _log_int(rng, 1, 4096), "rows": _log_int(rng, 100_000, 1_000_000)}
  if kind == "embedding":
    return {"kind": kind, "batch": _log_int(rng, 1000, 40000), "tables": rng.randint(1, 12),
            "rows": _log_int(rng, 10_000, 1_000_000), "dim": rng.choice([64, 128, 256]), "bag": _log_int(rng, 1, 40),
            "combiner": rng.choice(["sum", "mean", "sqrtn"]),
            "optimizer": rng.choice(["rowwise_adagrad", "adagrad", "adam"])}
  if kind == "hstu_train":
    mean = _log_int(rng, 40, 512)
    return {"kind": kind, "sequences": _log_int(rng, 8, 120), "mean_len": mean, "max_len": min(4096, mean * 8),
            "heads": rng.choice([1, 2, 4]), "layers": rng.randint(1, 8), "rows": _log_int(rng, 2000, 1_000_000),
            "negatives": rng.choice([32, 128, 512])}
  if kind == "hstu_encode":
    mean = _log_int(rng, 40, 512)
    return {"kind": kind, "sequences": _log_int(rng, 1, 120), "mean_len": mean, "max_len": min(4096, mean * 8),
            "heads": rng.choice([1, 2, 4]), "layers": rng.randint(1, 8)}
  if kind == "sasrec_train":
    return {"kind": kind, "batch": _log_int(rng, 32, 500), "length": rng.randint(50, 200),
            "rows": _log_int(rng, 10_000, 2_000_000)}
  if kind == "sasrec_eval":
    return {"kind": kind, "batch": _log_int(rng, 16, 512), "length": rng.randint(50, 200),
            "rows": _log_int(rng, 50_000, 1_000_000)}
  return {"kind": kind, "batch": _log_int(rng, 16, 250), "length": rng.randint(50, 256), "layers": rng.randint(1, 2)}


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed: int, device: str = DEVICE) -> torch.Generator:
  return torch.Generator(device=device).manual_seed(int(seed))


def _zipf(gen, vocab: int, n: int, alpha: float = 1.05) -> torch.Tensor:
  """`synthetic.zipf_ids` on the generator's device."""
  u = torch.rand(n, generator=gen, device=gen.device, dtype=torch.float64)
  a = 1.0 - alpha
  x = (((vocab + 1.0) ** a - 1.0) * u + 1.0) ** (1.0 / a)
  return (x.floor().long() - 1).clamp_(0, vocab - 1).to(torch.int32)


def _criteo_vocab(rows: int) -> tuple[int, ...]:
  return tuple(min(v, rows) for v in CRITEO_VOCAB)


def _dlrm_batch(gen, batch: int, vocab, bags) -> dict:
  dev = gen.device
  values = torch.cat([_zipf(gen, v, batch * b) for v, b in zip(vocab, bags)])
  lens = torch.tensor(bags, dtype=torch.int64, device=dev).repeat_interleave(batch)
  offsets = torch.zeros(lens.numel() + 1, dtype=torch.int32, device=dev)
  offsets[1:] = lens.cumsum(0)
  kjt = emb.KeyedJagged(tuple(f"cat_{i}" for i in range(len(vocab))), values, offsets, None, batch)
  dense = torch.log1p(torch.exp(torch.randn(batch, 13, generator=gen, device=dev)))
  label = (torch.rand(batch, generator=gen, device=dev) < 0.25).float()
  return {"dense": dense, "sparse": kjt, "label": label}


def _hstu_lengths(seed: int, c: dict) -> np.ndarray:
  """Power-law lengths of the case, in an order of the seed's own (the token count is the same for every seed)."""
  rng = np.random.default_rng(7)
  lens = synthetic.powerlaw_lengths(rng, c["sequences"], min(16, c["mean_len"] // 4), c["max_len"]).astype(np.float64)
  lens = np.clip(np.round(lens * c["mean_len"] / lens.mean()), 4, c["max_len"]).astype(np.int64)
  while lens.sum() > 1.5 * c["mean_len"] * c["sequences"]:
    lens[np.argmax(lens)] //= 2
  return np.random.default_rng(seed).permutation(lens)


def _timestamps(gen, lens: np.ndarray) -> torch.Tensor:
  gaps = torch.empty(int(lens.sum()), dtype=torch.float64, device=gen.device).exponential_(1.0 / 3600.0, generator=gen)
  return (1.6e9 + gaps.cumsum(0)).long()       # increasing inside every sequence; only differences matter


def _offsets(lens: np.ndarray) -> torch.Tensor:
  return torch.from_numpy(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)).to(DEVICE)


# ---- prepare -----------------------------------------------------------------------------------------------------
def _dense_moments(state) -> dict:
  """What the optimizer keeps of the step's gradients: the first moments (Adam) or the squared sums (Adagrad)."""
  opt = state.optimizer
  slot = "mu" if "mu" in opt.slots else "sum_of_squares"
  return {n: t for n, t in zip(opt.names, opt.slots[slot])}


def _tables(module) -> dict:
  out = {f"table{i}": w for i, w in enumerate(module.stack_weights)}
  for i, slots in enumerate(module.stack_slots):
    out.update({f"slot{i}.{n}": t for n, t in slots.items()})
  return out


def _warm_up(rate: float):
  """A rate that is zero while the step warms up and is captured."""
  return lambda step: rate if step >= 3 else 0.0


def _prepare_dlrm(c: dict, seed: int) -> dict:
  """The captured training step of `bench.py` (tiny: the small experiment's geometry and optimizer)."""
  if c["kind"] == "dlrm_tiny":
    d = c["dim"]
    vocab, bags = (c["rows"],) * c["tables"], (1,) * c["tables"]
    cfg = dlrm_experiment.ModelConfig(vocab_sizes=vocab, bag_sizes=bags, embedding_dim=d, bottom_mlp_dims=(64, d),
                                      top_mlp_dims=(64, 1), num_cross_layers=2, cross_rank=None,
                                      embedding_learning_rate=_warm_up(0.01), embedding_init_scale=0.01)
    opt = optim_factory.AdagradFactory(learning_rate=_warm_up(0.01))
  else:
    vocab, bags = _criteo_vocab(c["rows"]), CRITEO_BAGS
    cfg = dlrm_experiment.ModelConfig(vocab_sizes=vocab, bag_sizes=bags, embedding_learning_rate=_warm_up(0.004),
                                      embedding_init_scale=0.03)      # rows of the size training gives them
    opt = optim_factory.AdamFactory(learning_rate=_warm_up(2e-4))
  task = dlrm_experiment.PredictionTask(cfg, None, None, opt)
  part = partitioning.DataParallelPartitioner(use_cuda_graph=True, graph_warmup_steps=2)
  batch = _dlrm_batch(_gen(seed), c["batch"], vocab, bags)
  state = part.partition_init(lambda b: task.create_state(b, torch.Generator().manual_seed(seed)))(batch)
  rng = torch.Generator(device=DEVICE)
  step = part.partition_step(lambda inp, st: task.train_step(inp, st, rng), training=True)
  for _ in range(3):                            # two eager steps, then the capture and its first replay
    state, _ = step(batch, state)
  return {"case": c, "step": step, "state": state, "batch": batch}


def _prepare_predict(c: dict, seed: int) -> dict:
  vocab = _criteo_vocab(c["rows"])
  torch.manual_seed(seed)
  model = dlrm_model.DLRMDCNv2(vocab_sizes=vocab, bag_sizes=CRITEO_BAGS, device=torch.device(DEVICE), seed=seed)
  batch = _dlrm_batch(_gen(seed), c["batch"], vocab, CRITEO_BAGS)
  host = batch["sparse"]
  kjt = emb.KeyedJagged(host.keys, host.values.cpu(), host.offsets.cpu(), None, c["batch"])
  return {"case": c, "predictor": serving.Predictor(model), "batch": (batch["dense"].cpu(), kjt)}


def _prepare_embedding(c: dict, seed: int) -> dict:
  gen = _gen(seed)
  spec = {"rowwise_adagrad": emb.RowWiseAdagradOptimizerSpec, "adagrad": emb.AdagradOptimizerSpec,
          "adam": emb.AdamOptimizerSpec}[c["optimizer"]](learning_rate=0.01)
  names = tuple(f"f{i}" for i in range(c["tables"]))
  specs = {n: emb.EmbeddingSpec(c["rows"], c["dim"], combiner=c["combiner"], initializer=emb.specs.normal_init(0.05))
           for n in names}
  module = emb.ShardedEmbedding(emb.ShardedEmbeddingConfig(specs, spec, seed=seed % 100_000), device=DEVICE)
  # jagged bags: sizes geometric around the mean, empty ones among them
  n = c["tables"] * c["batch"]
  u = torch.rand(n, generator=gen, device=DEVICE).clamp_min_(1e-6)
  lens = (u.log() / math.log(c["bag"] / (c["bag"] + 1.0))).long().clamp_(0, 8 * c["bag"])
  offsets = torch.zeros(n + 1, dtype=torch.int32, device=DEVICE)
  offsets[1:] = lens.cumsum(0)
  values = _zipf(gen, c["rows"], int(lens.sum()))
  kjt = emb.KeyedJagged(names, values, offsets, None, c["batch"])
  grad = (torch.randn(c["batch"], c["tables"], c["dim"], generator=gen, device=DEVICE) * 0.1).to(torch.bfloat16)
  return {"case": c, "module": module.train(), "kjt": kjt, "grad": grad}


def _prepare_hstu_train(c: dict, seed: int) -> dict:
  gen = _gen(seed)
  lens = _hstu_lengths(seed, c)
  T = int(lens.sum())
  cfg = hstu_experiment.HSTUModelConfig(
      vocab_size=c["rows"], model_dim=64 * c["heads"], num_heads=c["heads"], num_layers=c["layers"],
      max_seq_len=c["max_len"], mean_seq_len=c["mean_len"], sequences_per_batch=c["sequences"],
      token_capacity=int(1.5 * c["mean_len"] * c["sequences"]) + 8, num_negatives=c["negatives"],
      num_in_batch=c["negatives"])
  task = hstu_experiment.HSTUTask(cfg, None)
  ids = _zipf(gen, c["rows"], T + 1)
  offsets = _offsets(lens)
  weights = torch.ones(T, device=DEVICE)
  weights[offsets[1:].long() - 1] = 0.0          # the last position of a sequence has no next item
  batch = {"input_ids": ids[:T].contiguous(), "target_ids": ids[1:].contiguous(), "seq_offsets": offsets,
           "negative_ids": torch.randint(0, c["rows"], (c["negatives"],), generator=gen, device=DEVICE).int(),
           "timestamps": _timestamps(gen, lens), "target_weights": weights}
  part = partitioning.DataParallelPartitioner()
  state = part.partition_init(lambda b: task.create_state(b, torch.Generator().manual_seed(seed)))(batch)
  rng = torch.Generator(device=DEVICE)
  step = part.partition_step(lambda inp, st: task.train_step(inp, st, rng), training=True)
  return {"case": c, "step": step, "state": state, "batch": batch}


def _prepare_hstu_encode(c: dict, seed: int) -> dict:
  gen = _gen(seed)
  lens = _hstu_lengths(seed, c)
  torch.manual_seed(seed)
  model = hstu_layers.HSTU(vocab_size=None, model_dim=64 * c["heads"], num_heads=c["heads"], num_layers=c["layers"],
                           use_relative_bias=True, max_seq_len=c["max_len"]).to(DEVICE).eval()
  e = torch.randn(int(lens.sum()), 64 * c["heads"], generator=gen, device=DEVICE).to(torch.bfloat16)
  return {"case": c, "model": model, "e": e, "offsets": _offsets(lens), "timestamps": _timestamps(gen, lens)}


def _sasrec_batch(gen, c: dict) -> dict:
  B, L = c["batch"], c["length"]
  lens = torch.randint(min(5, L), L + 1, (B,), generator=gen, device=DEVICE)
  seq = _zipf(gen, c["rows"] - 1, B * (L + 1), 1.1).view(B, L + 1) + 1          # id 0 is padding
  mask = torch.arange(L, device=DEVICE)[None, :] >= (L - lens)[:, None]          # right-aligned
  neg = torch.randint(1, c["rows"], (B, L), generator=gen, device=DEVICE).int()
  zero = torch.zeros((), dtype=torch.int32, device=DEVICE)
  return {"input_ids": torch.where(mask, seq[:, :L], zero), "positive_ids": torch.where(mask, seq[:, 1:], zero),
          "negative_ids": torch.where(mask, neg, zero), "padding_mask": mask.int()}


def _prepare_sasrec(c: dict, seed: int) -> dict:
  cfg = sasrec_experiment.SASRecConfig(vocab_size=c["rows"], max_positions=c["length"], batch_size=c["batch"])
  task = sasrec_experiment.SASRecTask(cfg, None)
  batch = _sasrec_batch(_gen(seed), c)
  part = partitioning.DataParallelPartitioner()
  state = part.partition_init(lambda b: task.create_state(b, torch.Generator().manual_seed(seed)))(batch)
  rng = torch.Generator(device=DEVICE)
  step = part.partition_step(lambda inp, st: task.train_step(inp, st, rng), training=True)
  return {"case": c, "step": step, "state": state, "batch": batch, "target": batch["positive_ids"][:, -1].long()}


def _prepare_mamba(c: dict, seed: int) -> dict:
  gen = _gen(seed)
  torch.manual_seed(seed)
  model = mamba_layers.Mamba2Stack(c["layers"], d_model=256, d_state=64, expand=2, nheads=8,
                                   ffn_expand=4).to(DEVICE).train()
  shape = (c["batch"], c["length"], 256)
  x = torch.randn(shape, generator=gen, device=DEVICE).to(torch.bfloat16).requires_grad_()
  lens = torch.randint(min(5, c["length"]), c["length"] + 1, (c["batch"],), generator=gen, device=DEVICE)
  mask = torch.arange(c["length"], device=DEVICE)[None, :] < lens[:, None]
  grad = (torch.randn(shape, generator=gen, device=DEVICE) * 0.1).to(torch.bfloat16)
  return {"case": c, "model": model, "x": x, "mask": mask, "grad": grad}


def prepare(case: dict, seed: int) -> dict:
  kind = case["kind"]
  if kind in ("dlrm_train", "dlrm_tiny"):
    return _prepare_dlrm(case, seed)
  return {"dlrm_predict": _prepare_predict, "embedding": _prepare_embedding, "hstu_train": _prepare_hstu_train,
          "hstu_encode": _prepare_hstu_encode, "sasrec_train": _prepare_sasrec, "sasrec_eval": _prepare_sasrec,
          "mamba_train": _prepare_mamba}[kind](case, seed)


# ---- run ---------------------------------------------------------------------------------------------------------
def run(s: dict):
  kind = s["case"]["kind"]
  if kind in ("dlrm_train", "dlrm_tiny", "hstu_train", "sasrec_train"):
    state, metrics = s["step"](s["batch"], s["state"])
    items = state.model.embedding if kind.startswith("dlrm") else state.model.items
    out = {"loss": metrics["loss"].total, "moments": _dense_moments(state), **_tables(items)}
    if kind == "dlrm_tiny":
      out["params"] = dict(state.params)
    return out
  if kind == "dlrm_predict":
    return s["predictor"].predict(s["batch"])
  if kind == "embedding":
    out = s["module"](s["kjt"])
    out.backward(s["grad"])
    return {"out": out, **_tables(s["module"])}
  if kind == "hstu_encode":
    with torch.no_grad():
      return s["model"].encode_jagged(s["e"], s["offsets"], s["timestamps"])
  if kind == "sasrec_eval":
    s["state"].model.eval()
    ranks = s["state"].model.evaluate_ranks(s["batch"]["input_ids"], s["batch"]["padding_mask"], s["target"])
    return ranks.float()                        # as the ranking metrics take them
  s["x"].grad = None
  s["model"].zero_grad(set_to_none=True)
  y = s["model"](s["x"], s["mask"])
  y.backward(s["grad"])
  return {"y": y, "dx": s["x"].grad, "grads": {n: p.grad for n, p in s["model"].named_parameters()}}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _distinct(vocab: int, n: float, alpha: float = 1.05) -> float:
  """Expected number of distinct ids among n Zipf draws."""
  r = np.unique(np.geomspace(1, vocab + 1, 4000).astype(np.int64))
  a = 1.0 - alpha
  lo, hi = r[:-1].astype(np.float64), r[1:].astype(np.float64)
  p = (hi ** a - lo ** a) / ((vocab + 1.0) ** a - 1.0) / (hi - lo)         # mean probability of a row in [lo, hi)
  return float(((hi - lo) * -np.expm1(n * np.log1p(-np.minimum(p, 1 - 1e-12)))).sum())


def _attention_pairs(c: dict) -> float:
  lens = _hstu_lengths(0, c).astype(np.float64)
  return float((lens * (lens + 1) / 2).sum())


def work(case: dict) -> dict:
  c, kind = case, case["kind"]
  if kind in ("dlrm_train", "dlrm_tiny", "dlrm_predict"):
    B = c["batch"]
    if kind == "dlrm_tiny":
      vocab, bags, d = (c["rows"],) * c["tables"], (1,) * c["tables"], c["dim"]
      bottom, top = [13, 64, d], [d * (1 + c["tables"]), 64, 1]
      cross = 2 * top[0] * top[0]
    else:
      vocab, bags, d = _criteo_vocab(c["rows"]), CRITEO_BAGS, 128
      bottom, top = [13, 512, 256, 128], [27 * 128, 1024, 1024, 512, 256, 1]
      cross = 3 * 2 * top[0] * 512
    weights = sum(a * b for dims in (bottom, top) for a, b in zip(dims, dims[1:])) + cross
    ids = B * sum(bags)
    rows = sum(_distinct(v, B * b) for v, b in zip(vocab, bags))
    read = ids * 4 + B * 14 * 4 + rows * d * 4
    if kind == "dlrm_predict":
      return {"bytes": read + weights * 2 + B * 4, "flops": 2.0 * B * weights + ids * d}
    moments = 2 if kind == "dlrm_train" else 1
    # rows and their accumulators read and written once, dense weights and optimizer state too
    return {"bytes": read + rows * (d * 4 + 8) + weights * (8 + 8 * moments),
            "flops": B * (6.0 * weights - 2.0 * bottom[0] * bottom[1]) + 3.0 * ids * d}
  if kind == "embedding":
    F, B, d = c["tables"], c["batch"], c["dim"]
    ids = F * B * c["bag"]
    rows = F * _distinct(c["rows"], B * c["bag"])
    slots = {"rowwise_adagrad": 8, "adagrad": 8 * d, "adam": 16 * d}[c["optimizer"]]
    return {"bytes": ids * 4 + F * B * (4 + 4 * d) + rows * (8 * d + slots), "flops": 3.0 * ids * d}
  if kind in ("hstu_train", "hstu_encode"):
    D, T, layers = 64 * c["heads"], float(_hstu_lengths(0, c).sum()), c["layers"]
    gemm, attn = layers * 2.0 * T * 5 * D * D, layers * 4.0 * _attention_pairs(c) * D
    if kind == "hstu_encode":
      return {"bytes": T * (4 * D + 8) + layers * 5 * D * D * 2, "flops": gemm + attn}
    rows = _distinct(c["rows"], T) + c["negatives"]
    logits = 2.0 * T * 2 * c["negatives"] * D
    return {"bytes": T * 24 + rows * (8 * D + 8) + layers * 5 * D * D * 24,
            "flops": 3 * gemm + 2.5 * attn + attn + 3 * logits}
  if kind in ("sasrec_train", "sasrec_eval"):
    B, D, L = c["batch"], 256, c["length"]
    T = B * (5 + L) / 2.0                       # real tokens
    weights = 2 * (4 * D * D + 2 * 1024 * D)
    gemm, attn = 2.0 * T * weights, 2 * 4.0 * D * B * (L * L / 6.0)
    if kind == "sasrec_eval":
      return {"bytes": c["rows"] * D * 4.0 + T * 4 + B * 16, "flops": gemm + attn + 2.0 * B * c["rows"] * D}
    rows = _distinct(c["rows"], T, 1.1) + min(T, c["rows"])
    return {"bytes": T * 16 + rows * (8 * D + 8) + weights * 24.0, "flops": 3 * gemm + 3.5 * attn + 9 * T * D}
  B, L, D = c["batch"], c["length"], 256
  T = float(B * L)
  weights = D * (2 * 512 + 128 + 8) + 512 * D + 2 * 4 * D * D
  scan = 2.0 * T * 512 * 64 * 2                  # state update and read-out of every head
  return {"bytes": T * D * 2 * 4 + c["layers"] * weights * 8.0, "flops": 3 * c["layers"] * (2.0 * T * weights + scan)}


def tolerance(case: dict) -> dict:
  """Relative errors between formulations of equal precision (other summation orders, other places of the same bf16
  roundings): about four times what two passes over the kernels and over fp32 library products of the same bf16
  operands differ by (DLRM steps: 0.9 % and 0.24 of the mean square root, for the gradients of the cross layers).  The
  DLRM and retrieval steps normalise tiny per-row gradients, so single elements move by a large part of the mean."""
  return {
      "dlrm_train": {"rel": 3e-2, "max": 0.9}, "dlrm_tiny": {"rel": 1e-4, "max": 1e-2},
      "dlrm_predict": {"rel": 2.5e-2, "max": 0.12}, "embedding": {"rel": 1e-4, "max": 3e-2},
      "hstu_train": {"rel": 3e-2, "max": 0.9}, "hstu_encode": {"rel": 2.5e-2, "max": 0.16},
      "sasrec_train": {"rel": 1.5e-2, "max": 0.4}, "sasrec_eval": {"rel": 7e-3, "max": 3e-2},
      "mamba_train": {"rel": 1.6e-2, "max": 0.2},
  }[case["kind"]]
