"""Workloads that the framework's speed is judged on, and how to run one pass of each.

Five kinds of pass, each through the call that the training command itself makes:

  step   ``Trainer.train_step``: a whole optimiser step from host batches (microbatches, AdamW, DiLoCo outer step)
  train  ``forward_backward`` of the stage that owns the loss, one microbatch, gradients added to the main gradient
  stage  ``forward`` and ``backward`` of a pipeline stage in front of it, one microbatch
  eval   ``forward_loss``, one microbatch of an evaluation
  infer  ``forward_infer``, one position of the sampling loop (it runs the whole sequence per token)

Models are those of ``configs/model`` cut into equal pipeline stages, and the two-layer model of the tests;
microbatch sizes and sequence lengths run from one short sentence to the largest microbatch of ``experiments/``.
"""
import itertools
import math
import os
import tempfile

import torch

from diloco_swarm_b200.config import Config
from diloco_swarm_b200.models.engine_b200 import B200Engine
from diloco_swarm_b200.models.gpt2 import GPT2Config, split_layers, stage_param_specs
from diloco_swarm_b200.train import Trainer
from diloco_swarm_b200.world import World

# layers, heads, width, vocabulary, longest sequence
MODELS = {
    "test": (2, 4, 128, 512, 128),
    "gpt2-tiny": (4, 4, 128, 50304, 1024),
    "gpt2-small": (12, 12, 768, 50304, 1024),
    "gpt2-medium": (24, 16, 1024, 50304, 1024),
    "gpt2-large": (36, 20, 1280, 50304, 1024),
    "gpt2-xl": (48, 25, 1600, 50304, 1024),
}
USED_IDS = 50257          # the tokenizer fills this much of the padded vocabulary


def case(name, kind, model, batch, seq, stages=1, stage=0, **more):
    """``batch`` sequences of ``seq`` tokens per microbatch on stage ``stage`` of ``stages``.

    ``padded``: sequences end early and the rest is masked out of the loss; ``chunks``: slices of the LM head;
    ``tied``: head and embedding share their weights; ``micros``: microbatches per optimiser step; ``outer``:
    a DiLoCo outer step ends the step."""
    c = {"kind": kind, "model": model, "batch": batch, "seq": seq, "stages": stages, "stage": stage, "padded": False,
         "chunks": 1, "tied": False, "micros": 1, "outer": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # sampling during a memorisation run: five samples of the four-character prompt plus twenty new tokens
        case("sample-tiny", "infer", "gpt2-tiny", 5, 24),
        # the same on the model that the experiments train
        case("sample-small", "infer", "gpt2-small", 5, 24),
        # sampling towards the end of a long continuation
        case("sample-small-long", "infer", "gpt2-small", 8, 777),
        # the memorisation smoke run: two microbatches of one padded sentence, then AdamW
        case("step-tiny", "step", "gpt2-tiny", 1, 128, micros=2, padded=True),
        # the model-size sweep's smallest model at its microbatch of 64: nearly all of it is the LM head
        case("train-tiny", "train", "gpt2-tiny", 64, 1024),
        # short padded text examples on the experiments' model, a length that no tile divides
        case("train-small-short", "train", "gpt2-small", 16, 133, padded=True),
        # the SWARM experiments' microbatch of 32 full sequences: the largest case
        case("train-small", "train", "gpt2-small", 32, 1024),
        # a DiLoCo step of the headline configuration (microbatch 16) with fewer microbatches than its 32
        case("step-small", "step", "gpt2-small", 16, 1024, micros=2, outer=True),
        # evaluation of the experiments' model
        case("eval-small", "eval", "gpt2-small", 32, 1024),
        # a middle stage of the medium model on four stages (microbatch 8 as in the model-size sweep)
        case("stage-medium", "stage", "gpt2-medium", 8, 1024, 4, 1),
        # the first stage of the large model (embedding and blocks, microbatch 4)
        case("stage-large", "stage", "gpt2-large", 4, 1024, 9, 0),
        # the last stage of the xl model (blocks, LM head, loss) on text of a thousand tokens
        case("train-xl", "train", "gpt2-xl", 2, 1000, 24, 23, padded=True),
    ]


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "stage", "stage", "eval", "infer", "infer", "step"])
        model = rng.choice(list(MODELS))
        layers, _, _, _, longest = MODELS[model]
        stages = rng.choice([s for s in (1, 2, 3, 4, 6, 8, 9, 12, 16, 24) if layers % s == 0])
        if kind in ("infer", "step"):
            stages = 1
        if kind == "stage":
            if stages == 1:
                continue
            stage = rng.randrange(stages - 1)
        else:
            stage = stages - 1
        seq = int(round(math.exp(rng.uniform(math.log(16), math.log(longest)))))
        if rng.random() < 0.5:
            seq = rng.choice([s for s in (64, 128, 256, 384, 512, 768, 1024) if s <= longest])
        batch = int(round(math.exp(rng.uniform(0, math.log(64)))))
        c = case(None, kind, model, batch, seq, stages, stage, padded=rng.random() < 0.4)
        if kind == "train" and rng.random() < 0.2:
            c["chunks"] = rng.choice([2, 4])
        if stages == 1 and rng.random() < 0.15:
            c["tied"] = True
        if kind == "step":
            c["micros"], c["outer"] = rng.choice([1, 2, 3, 4]), rng.random() < 0.5
        # what one GPU holds three times over, quick to prepare, and no larger than the largest listed case
        if parameters(c) > 2.2e8 or work(c)["flops"] > most or (kind == "infer" and batch * seq > 8192):
            continue
        return c


def config_of(c):
    layers, heads, width, vocab, longest = MODELS[c["model"]]
    return GPT2Config(block_size=longest, vocab_size=vocab, n_layer=layers, n_head=heads, n_embd=width,
                      parameter_sharing=c["tied"])


def specs_of(c):
    """(key, name, shape) of the stage's tensors."""
    g = config_of(c)
    layers = split_layers(g.n_layer, c["stages"])[c["stage"]]
    return stage_param_specs(g, layers, c["stage"] == 0, c["stage"] == c["stages"] - 1)


def parameters(c):
    return sum(math.prod(shape) for _, _, shape in specs_of(c))


def work(c):
    layers, _, d, vocab, _ = MODELS[c["model"]]
    n, tokens, seq = layers // c["stages"], c["batch"] * c["seq"], c["seq"]
    head = c["stage"] == c["stages"] - 1
    matmul = 2.0 * tokens * (n * 12 * d * d + (vocab * d if head else 0))
    attention = 2.0 * tokens * seq * d * n                # Q K^T and P V under the causal mask
    params = parameters(c)
    # of an embedding table that is not the head as well, only the rows in use are touched
    dense = params - (vocab * d if c["stage"] == 0 and not (head and c["tied"]) else 0)
    ends = 8.0 * tokens if c["stage"] == 0 else 2.0 * tokens * d
    if c["kind"] == "infer":
        return {"flops": matmul + attention, "bytes": 2.0 * dense + ends + 4.0 * tokens * vocab}
    if c["kind"] == "eval":
        return {"flops": matmul + attention, "bytes": 2.0 * dense + ends + 16.0 * tokens}
    ends = 2 * ends + (16.0 * tokens if head else 4.0 * tokens * d)
    one = {"flops": 3 * matmul + 3.5 * attention, "bytes": 10.0 * dense + ends}
    if c["kind"] != "step":
        return one
    # weights, gradient and both moments in, all of them and the bf16 weights out; the outer step's weights and momentum
    update = params * (34.0 + (26.0 if c["outer"] else 0.0))
    return {"flops": c["micros"] * one["flops"], "bytes": c["micros"] * one["bytes"] + update}


def tolerance(c):
    """Activations and their gradients are rounded to bf16 some eight times per block and direction.  One rounding
    is off by about 1.1e-3 of the value (uniform within half a unit of the eighth bit), and independent ones add
    up in squares; two implementations at this precision differ by that, and by 1e-2 in any case."""
    blocks = MODELS[c["model"]][0] // c["stages"]
    directions = 1 if c["kind"] in ("infer", "eval") else 2
    rel = max(1e-2, 1.1e-3 * math.sqrt(8 * directions * blocks))
    if c["kind"] == "step":
        rel = max(rel, 2e-2)                              # the second moment is the gradient's square
    return {"rel": rel, "max": 0.5}


# ---------------------------------------------------------------------- engines
# An engine outlives its batches: a program builds one and feeds it for days.  So engines are kept when the state
# that used them goes away, and the next state of the same configuration gets fresh weights in the same buffers.
# Buffers that peers can map are not returned to the allocator by garbage collection, so an engine of another
# configuration is closed before a new one is built.
_idle = {}
_runs = itertools.count()


def engine_key(c):
    key = [c["model"], c["stages"], c["stage"], c["tied"], c["chunks"]]
    return tuple(key + [c["kind"], c["batch"], c["seq"], c["micros"], c["outer"]]) if c["kind"] == "step" else tuple(key)


def build(c):
    """A ``Trainer`` for whole steps, else the stage's engine."""
    layers, heads, width, vocab, longest = MODELS[c["model"]]
    outer = {"type": "SGD", "lr": 0.7, "momentum": 0.9, "nesterov": True} if c["outer"] else {"type": "None", "lr": 0.0}
    config = Config(
        model={"n_layer": layers, "n_head": heads, "n_embd": width, "vocab_size": vocab, "block_size": longest,
               "parameter_sharing": c["tied"]},
        data={"path": "synthetic:zipf", "seq_length": c["seq"]},
        train={"micro_batch_size": c["batch"], "batch_size": c["batch"] * c["micros"], "lm_head_chunks": c["chunks"],
               "inner_optimizer": {"type": "AdamW", "lr": 4e-4}, "outer_optimizer": outer},
        swarm={"num_stages": c["stages"], "sync_every_n_steps": 1},
        eval={"enable": False}, sample={"enable": False},
        logging={"log_dir": os.path.join(tempfile.gettempdir(), "dswarm_cases"), "run_id": f"{os.getpid()}-{next(_runs)}",
                 "console": {"log_level": "ERROR"}, "file": {"log_level": "ERROR"}})
    world = World(1, device_type="cuda", init=False)
    device = torch.device("cuda", torch.cuda.current_device())
    if c["kind"] == "step":
        made = Trainer(config, world=world)
        made.num_train_steps = 1000
        return made
    world.num_stages, world.stage = c["stages"], c["stage"]
    return B200Engine(config_of(c), world, config, device)


def engine_of(made):
    return made.engine if isinstance(made, Trainer) else made


class State:
    """What a training program holds: the engine (and its trainer) and one microbatch or batch."""

    def __init__(self, c):
        self.case, self.key, self.steps = dict(c), engine_key(c), 0
        for key in [k for k in _idle if k != self.key]:
            for made in _idle.pop(key):
                torch.cuda.synchronize()
                for buf in engine_of(made).symmetric_buffers():
                    buf.close()
                if isinstance(made, Trainer):
                    made.logger.close()
        self.made = _idle[self.key].pop() if _idle.get(self.key) else build(c)
        self.engine = engine_of(self.made)

    def __del__(self):
        if getattr(self, "made", None) is not None:
            _idle.setdefault(self.key, []).append(self.made)


def zipf_ids(c, gen):
    """Token ids with the frequencies of text (Zipf), one more per sequence than the model reads."""
    used = min(USED_IDS, MODELS[c["model"]][3])
    cdf = torch.arange(1, used + 1, dtype=torch.float64, device=gen.device).reciprocal().cumsum(0)
    u = torch.rand(c["batch"] * c["micros"], c["seq"] + 1, generator=gen, device=gen.device, dtype=torch.float64)
    return torch.searchsorted(cdf, u * cdf[-1]).clamp_(max=used - 1)


def prepare(c, seed):
    state = State(c)
    eng = state.engine
    dev = eng.device
    gen = torch.Generator(device=dev).manual_seed(int(seed))

    def normal(*shape, std=1.0, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32).mul_(std).to(dtype)

    weights = {}
    for key, name, shape in specs_of(c):
        std = 0.02 / math.sqrt(2 * MODELS[c["model"]][0]) if name.endswith("c_proj.weight") else 0.02
        weights[key] = normal(*shape, std=std)
        if len(shape) == 1 and name.endswith("weight"):
            weights[key] += 1.0                           # LayerNorm gains
    eng.load_state_dict(weights)
    del weights
    # moments of a run that is under way (at the first step Adam's update is the gradient's sign, noise where it is small)
    eng.load_optim_state({"m": normal(eng.n, std=3e-5), "v": (normal(eng.n, std=1e-4).abs() + 5e-5).square(), "opt_step": 1000})
    eng.grad.zero_()
    eng.reset_outer()
    eng.train() if c["kind"] in ("step", "train", "stage") else eng.eval()

    tokens = zipf_ids(c, gen)
    rows, seq, d = tokens.shape[0], c["seq"], eng.cfg.n_embd
    mask = torch.ones(rows, seq, dtype=torch.long, device=dev)
    if c["padded"]:
        length = torch.randint(max(1, seq // 4), seq + 1, (rows, 1), generator=gen, device=dev)
        mask = (torch.arange(seq, device=dev) < length).long()
    batch = {"input_ids": tokens[:, :-1].contiguous(), "target_ids": tokens[:, 1:].contiguous(), "attention_mask": mask}
    if c["kind"] == "step":
        state.made.opt_steps = 0
        state.batch = {k: v.cpu().pin_memory() for k, v in batch.items()}
        return state
    state.batch = batch
    state.ids = batch["input_ids"] if c["stage"] == 0 else None
    # hidden states and gradients as a neighbouring stage sends them
    state.hidden = None if c["stage"] == 0 else normal(rows, seq, d, dtype=torch.bfloat16)
    state.grad_out = normal(rows, seq, d, std=1e-3, dtype=torch.bfloat16) if c["kind"] == "stage" else None
    return state


def run(state):
    c, eng, b = state.case, state.engine, state.batch
    if c["kind"] == "infer":
        return eng.forward_infer(state.ids, state.hidden)
    if c["kind"] == "eval":
        return eng.forward_loss(state.ids, state.hidden, b["target_ids"], b["attention_mask"], 1.0)
    if c["kind"] == "train":
        loss, dx = eng.forward_backward(0, state.ids, state.hidden, b["target_ids"], b["attention_mask"], 1.0)
        return {"loss": loss, "dx": dx, "grad": eng.grad}
    if c["kind"] == "stage":
        y = eng.forward(0, state.ids, state.hidden)
        dx = eng.backward(0, state.grad_out)
        return {"y": y, "dx": dx, "grad": eng.grad}
    state.steps += 1
    out, _ = state.made.train_step(state.steps, b)
    got = {"loss": out.loss, "norm": out.norm, "weights": eng.theta, "bf16": eng.w16, "m": eng.m, "v": eng.v}
    if eng.outer is not None:
        got["global"], got["momentum"] = eng.outer.theta_g, eng.outer.mom
    return got
