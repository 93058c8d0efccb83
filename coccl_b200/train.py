"""Training engine: micro-batch loop, (optional) pipeline schedule, sharded optimizer.

`Trainer.train_step(tokens)` is the public entry point used by bench.py and the
examples: it takes one global-batch slice of token ids for this data-parallel
rank as a pinned host tensor [sequences, seq_len + 1], copies it to the device,
runs forward/backward over all micro-batches, reduces gradients, steps the
optimizer and returns the mean loss as a device scalar.
"""
from __future__ import annotations

import operator
import warnings
from dataclasses import dataclass

import torch

from . import _lib
from .models.gpt import GPTConfig, GPTStage, NoTP, ParamStore, TransformerLayer
from .parallel.dp import DistributedOptimizer


@dataclass
class ParallelConfig:
    tp: int = 1
    pp: int = 1
    dp: int = 1
    sequence_parallel: bool = True
    # "zero1": sharded optimizer (reduce-scatter + all-gather); "ddp": gradient all-reduce; "fsdp": parameters, gradients
    # and optimizer state all sharded, a layer's parameters gathered while it runs (data parallelism only)
    dp_strategy: str = "zero1"
    ep: int = 1   # expert parallelism of a mixture-of-experts model: 1 (every rank holds all experts) or dp
    virtual_stages: int = 1   # model chunks per pipeline rank; > 1 selects the interleaved 1F1B schedule
    cp: int = 1   # context parallelism: ranks that share every sequence, each holding seq_len / cp positions of it


def split_layers(n_layer: int, stages: int) -> list[tuple[int, int]]:
    """Layer range [first, last) of each of `stages` consecutive (virtual) pipeline stages. Layers that do not divide
    evenly go to the FIRST stages: the last one also runs the final LayerNorm, the output head and the loss, which cost
    about one transformer layer (2 * hidden * vocab against 24 * hidden^2 FLOPs per token for GPT-6.7B)."""
    assert 1 <= stages <= n_layer, f"{n_layer} layers cannot fill {stages} pipeline stages"
    base, extra = divmod(n_layer, stages)
    out, first = [], 0
    for s in range(stages):
        n = base + (1 if s < extra else 0)
        out.append((first, first + n))
        first += n
    return out


def _own_code() -> list:
    """(namespace, look-up of names in it, what it finds) of the functions, classes and methods that a pass through a stage can
    reach by name, as this package and PyTorch define them."""
    from torch.nn.modules import module as nnm
    from .models import gpt, llama
    from .ops import fused, gemm
    own = (gpt.GPTStage, gpt.TransformerLayer, gpt.NoTP, gpt.GPTConfig, llama.LlamaLayer, Trainer, fused._Linear, fused._LayerNorm,
           fused._RmsNorm, fused._RotateQkv, fused._Swiglu, fused._Embed, fused._CrossEntropy)
    spaces = [(vars(x), [k for k, v in vars(x).items() if callable(v) or isinstance(v, (staticmethod, classmethod, property))])
              for x in (gpt, llama, fused, gemm, _lib, *own)]
    spaces += [(vars(torch.nn.functional), ["scaled_dot_product_attention", "embedding", "silu"]), (vars(nnm.Module), ["__call__", "_call_impl"]),
               (vars(torch.Tensor), ["backward"]), (vars(torch.autograd), ["backward"])]
    return [(ns, operator.itemgetter(*keys), operator.itemgetter(*keys)(ns)) for ns, keys in spaces if keys]


def _own_code_in_place() -> bool:
    try:
        return all(get(ns) == was for ns, get, was in _OWN_CODE)   # of functions and classes: by identity
    except KeyError:
        return False


class _Snapshot:
    """Everything a pass through a stage looks up in its modules, as it stood: their attributes, parameters and sub-modules, the
    fields of the objects they hold (configuration, tensor-parallel context), the elements of lists. Taken and compared by
    identity, and what is compared is kept alive, so that a new object can never pass for the old one."""

    # hook tables of a module: their identity is compared, what is in them is MicroBatchGraph._plain_context's to look at
    HOOKS = set(vars(torch.nn.Module())) - {"_parameters", "_buffers", "_modules"}

    def __init__(self, *roots):
        self.roots, self.parts, seen = roots, [], set()
        for r in roots:
            self._walk(r, seen)

    def _walk(self, obj, seen):
        if id(obj) in seen or isinstance(obj, (type, torch.Tensor, ParamStore)):
            return
        seen.add(id(obj))
        module = isinstance(obj, torch.nn.Module)
        if module or (type(obj).__module__.startswith(__package__) and hasattr(obj, "__dict__")):
            obj = obj.__dict__
        if isinstance(obj, dict):
            self.parts.append((obj.values(), [*obj.values()], obj, [*obj]))
            for k, v in obj.items():
                if not (module and k in self.HOOKS):
                    self._walk(v, seen)
        elif isinstance(obj, (list, tuple)):
            self.parts.append((obj, [*obj], (), []))
            for v in obj:
                self._walk(v, seen)

    def holds(self, *roots) -> bool:
        if not all(map(operator.is_, roots, self.roots)):
            return False
        for values, were, keys, named in self.parts:
            if len(values) != len(were) or not all(map(operator.is_, values, were)) or [*keys] != named:
                return False
        return True


_shape_of, _type_of, _trains = map(operator.attrgetter, ("shape", "dtype", "requires_grad"))


class MicroBatchGraph:
    """Forward and backward of one micro-batch as a CUDA graph, for models whose kernels are shorter than the host code that
    launches them, with the parameters' gradients as a branch of their own beside the backward pass (`fused.Branch`).

    A micro-batch is about 35 launches a layer through autograd, 1.2 ms of host time a layer; below that much device work a
    layer the GPU waits (2 layers 512 wide, two micro-batches of 512 tokens: 5.0 ms a step for 1.4 ms of kernels). Replayed,
    the launches cost the device only. Large models gain nothing and would keep a micro-batch's activations in the graph's
    pool, so the rule is on size (`worth_it`). A graph is captured when a step has been seen twice with nothing changed, so
    first steps on new inputs run as ever; it holds what its kernels address (the scratch buffers and tables as they were).

    A replay runs the kernels and none of the Python around them, so it stands in for a step only while that Python could not
    have done anything else: the stage is built of this package's own dense layers, whose methods and functions are the
    package's own; nothing the pass looks up has changed since the capture (`_Snapshot`), nor the buffers behind the parameters
    and their gradients, nor PyTorch's switches for attention, matrix products and determinism; and no hook, mode or context
    around the call would see the pass. Anything else goes back to the launches. Setting `enabled` to False does so for good,
    and gives the graph's memory back at the next step."""

    MAX_TOKENS = 16384
    MAX_LAYER_FLOPS = 1.5e12    # 1.1 ms at the 1.37 PFLOP/s of sustained bf16 products, against 1.2 ms of host time
    MAX_POOL_BYTES = 1 << 30    # the graph keeps the activations of a micro-batch beside the allocator's cache

    def __init__(self):   # no reference to the trainer: the two would keep each other's device memory until a collection
        self.enabled = True
        self._drop()

    def _drop(self):
        self.key = self.snapshot = self.sdp_order = self.seen = self.graph = self.tokens = self.keep = None
        self.launches = 0

    @classmethod
    def pool_bytes(cls, cfg: GPTConfig, n_tokens: int, branch: bool) -> float:
        # bf16 values a token leaves behind: 12 rows of the hidden size and 4 of the MLP's a layer, and its logits; with the
        # gradients that a branch of the backward pass reads, 6 and 2 more
        rows = (18 * cfg.hidden + 6 * cfg.ffn) if branch else (12 * cfg.hidden + 4 * cfg.ffn)
        return 2.0 * n_tokens * (cfg.n_layer * rows + cfg.vocab)

    @classmethod
    def worth_it(cls, cfg: GPTConfig, n_tokens: int) -> bool:
        return (n_tokens <= cls.MAX_TOKENS and cfg.flops_per_token() * n_tokens <= cls.MAX_LAYER_FLOPS * max(1, cfg.n_layer) and
                cls.pool_bytes(cfg, n_tokens, False) <= cls.MAX_POOL_BYTES)

    @staticmethod
    def own_code(stage) -> bool:
        """Whether `stage` is built of this package's own dense modules and single-GPU context, none of their methods replaced."""
        from .models.llama import LlamaLayer
        parts = [*stage.modules(), *(m.tp for m in stage.modules() if hasattr(m, "tp"))]
        return type(stage) is GPTStage and all(
            type(m) in (GPTStage, TransformerLayer, LlamaLayer, torch.nn.ModuleList, NoTP) and
            not any(callable(getattr(type(m), k, None)) for k in vars(m)) for m in parts)

    @staticmethod
    def _plain_context(stage) -> bool:
        """Nothing around the call that would want to see the forward and backward pass happen."""
        from torch.nn.modules import module as nnm
        hooked = any(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks for m in stage.modules())
        return (torch.is_grad_enabled() and not torch.is_autocast_enabled() and not torch.is_anomaly_enabled() and
                not torch.cuda.is_current_stream_capturing() and not hooked and not nnm._has_any_global_hook() and
                torch._C._len_torch_dispatch_stack() == 0 and torch._C._len_torch_function_stack() == 0 and
                torch._C._autograd._top_saved_tensors_default_hooks(True) is None)

    @staticmethod
    def _key(t, shape, scale):
        """What is compared by value; None where hooks on a parameter would see its gradient, or it has no gradient buffer."""
        from .ops import gemm as G
        sdp, cudnn, mm = torch.backends.cuda, torch.backends.cudnn, torch.backends.cuda.matmul
        switches = (sdp.flash_sdp_enabled(), sdp.mem_efficient_sdp_enabled(), sdp.math_sdp_enabled(), sdp.cudnn_sdp_enabled(),
                    sdp.fp16_bf16_reduction_math_sdp_allowed(),
                    torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled(),
                    torch.utils.deterministic.fill_uninitialized_memory, cudnn.enabled, cudnn.deterministic, cudnn.benchmark,
                    torch.get_float32_matmul_precision(), mm.allow_bf16_reduced_precision_reduction,
                    torch.get_default_dtype(), torch.is_inference_mode_enabled())
        params = [p for m in t.stage.modules() for p in m._parameters.values() if p is not None]
        grads = [getattr(p, "main_grad", None) for p in params]
        if any([p._backward_hooks or p._post_accumulate_grad_hooks for p in params]) or any([g is None for g in grads]):
            return None
        buffers = [*map(torch.Tensor.data_ptr, params), *map(torch.Tensor.data_ptr, grads), *map(_shape_of, params),
                   *map(_type_of, grads), *map(_trains, params)]
        return tuple(shape), scale, G.get_variant(), torch.cuda.current_device(), t._loss_acc.data_ptr(), switches, buffers

    def ready(self, t: "Trainer", shape, scale) -> bool:
        """Whether trainer t's micro-batches of this step are to be replayed (captures the graph at the third equal step)."""
        if not self.enabled:
            self._drop()
            return False
        if not (torch.device(t.device).type == "cuda" and t.schedule is None and t.groups is None and not t.fsdp and
                t.cfg.n_experts == 0 and self.worth_it(t.cfg, shape[0] * (shape[1] - 1)) and
                self._plain_context(t.stage) and "_micro_batch" not in vars(t) and type(t)._micro_batch is Trainer._micro_batch and
                _own_code_in_place()):
            return False
        key = self._key(t, shape, scale)
        if key is None:
            return False
        order = torch._C._get_sdp_priority_order()   # PyTorch fills it in at its first attention call
        if key != self.key or (self.graph is not None and not (self.snapshot.holds(t.stage, t.cfg) and order == self.sdp_order)):
            self._drop()
            self.key, self.seen = key, 1
            return False
        if self.graph is None:
            self.seen += 1
            if self.seen > 2 and self.own_code(t.stage):
                self.snapshot, self.sdp_order = _Snapshot(t.stage, t.cfg), order
                self._capture(t, shape, scale)
        return self.graph is not None

    def _give_up(self, why: str):
        self.enabled = False
        self._drop()
        warnings.warn(f"micro-batches of this trainer are launched kernel by kernel: {why}")

    def _capture(self, t, shape, scale):
        from .models import llama
        from .ops import fused, gemm
        params = list(t.stage.parameters())
        if any(p.grad is not None for p in params):
            return
        tokens = torch.zeros(tuple(shape), dtype=torch.int64, device=t.device)
        graph, side, cur = torch.cuda.CUDAGraph(), torch.cuda.Stream(t.device), torch.cuda.current_stream(t.device)
        before = _lib.lib().cocclkLaunchCount()
        side.wait_stream(cur)
        try:
            with torch.cuda.stream(side):
                graph.capture_begin(capture_error_mode="thread_local")
                try:
                    if self.pool_bytes(t.cfg, shape[0] * (shape[1] - 1), True) <= self.MAX_POOL_BYTES:
                        with fused.Branch(t.device):
                            t._micro_batch(tokens, scale)
                    else:
                        t._micro_batch(tokens, scale)
                finally:
                    graph.capture_end()
            if any(p.grad is not None for p in params):
                self._give_up("autograd leaves a gradient in `.grad`, which only the capture would see")
                return
        except RuntimeError as e:   # nothing has run: the launches take over
            self._give_up(f"the capture of the CUDA graph failed ({e})")
            return
        finally:
            cur.wait_stream(side)
            for p in params:
                p.grad = None
        self.graph, self.tokens = graph, tokens
        self.launches = _lib.lib().cocclkLaunchCount() - before
        self.keep = (list(fused._scratch.values()), list(gemm._err_words.values()), list(llama._ROPE_CACHE.values()))

    def run(self, mb):
        self.tokens.copy_(mb)
        self.graph.replay()
        _lib.lib().cocclkCountLaunches(self.launches)


class Trainer:
    def __init__(self, cfg: GPTConfig, device, *, micro_batch=2, parallel: ParallelConfig | None = None, groups=None,
                 lr=1e-4, weight_decay=0.1, clip_grad=1.0, seed=1234):
        self.cfg, self.device, self.micro_batch = cfg, device, micro_batch
        self.parallel = parallel or ParallelConfig()
        self.groups = groups  # coccl_b200.parallel.mesh.Mesh or None (single GPU)
        g = groups
        tp_ctx = g.tp_context() if g is not None else None
        pp_rank = g.pp_rank if g is not None else 0
        pp = self.parallel.pp
        chunks = self.parallel.virtual_stages if pp > 1 else 1
        assert chunks >= 1
        # virtual stage c * pp + pp_rank is this rank's chunk c (one chunk: the plain contiguous split)
        stages = split_layers(cfg.n_layer, pp * chunks)
        ranges = [stages[c * pp + pp_rank] for c in range(chunks)]
        dp = self.parallel.dp
        cp = self.parallel.cp
        assert cp == (g.cp if g is not None else 1), "ParallelConfig.cp and the mesh disagree"
        assert cfg.seq_len % cp == 0, "the sequence length must divide by the context-parallel size"
        self.cp_ctx = g.cp_context() if (g is not None and cp > 1) else None
        replicas = dp * cp   # ranks that hold the same parameters: the gradient / optimizer-shard group
        ep_comm = getattr(g, "ep_comm", None) if g is not None else None
        assert self.parallel.ep == (ep_comm.size if ep_comm is not None else 1), "ParallelConfig.ep and the mesh disagree"
        self.fsdp = self.parallel.dp_strategy == "fsdp"
        if self.fsdp:
            assert self.parallel.tp == pp == cp == self.parallel.ep == 1 and cfg.n_experts == 0, \
                "the fully sharded strategy is built for pure data parallelism of dense models"
        self.stage = GPTStage(cfg, device, tp=tp_ctx, layer_ranges=ranges, fsdp=self.fsdp,
                              fsdp_comm=(g.dp_comm if (g is not None and dp > 1) else None),
                              pre=(pp_rank == 0), post=(pp_rank == pp - 1), seed=seed, pad_to=8 * replicas * 2048,
                              ep_comm=ep_comm, cp=self.cp_ctx)
        # experts spread over the expert-parallel group: updated locally (never reduced or gathered), clipped with
        # the same coefficient as everything else; their squares enter the global norm through the main optimizer
        self.expert_opt = None
        es = self.stage.expert_store
        if es is not None:
            self.expert_opt = DistributedOptimizer(es.flat_param, es.flat_grad, None, lr=lr, weight_decay=weight_decay,
                                                   clip_grad=clip_grad)
        if self.fsdp:
            from .parallel.dp import FsdpOptimizer
            self.opt = FsdpOptimizer(self.stage.store, g.dp_comm if (g is not None and dp > 1) else None, lr=lr,
                                     weight_decay=weight_decay, clip_grad=clip_grad)
        norm_groups = []
        if g is not None:
            if g.tp_comm is not None and g.tp_comm.size > 1:
                norm_groups.append(g.tp_comm)
            if g.pp_comm is not None and g.pp_comm.size > 1:
                norm_groups.append(g.pp_comm)
        self.opt = self.opt if self.fsdp else DistributedOptimizer(self.stage.store.flat_param, self.stage.store.flat_grad,
                                        g.dp_comm if (g is not None and replicas > 1) else None, lr=lr,
                                        weight_decay=weight_decay, clip_grad=clip_grad, norm_groups=norm_groups,
                                        norm_exclude=self.stage.store.norm_exclude_ranges(
                                            g.tp_rank if g is not None else 0,
                                            drop_wte=(pp > 1 and pp_rank == pp - 1 and cfg.tie_embeddings)),
                                        extra_sumsq=(self.expert_opt.local_sum_squares if self.expert_opt is not None else None),
                                        strategy=self.parallel.dp_strategy)
        self.schedule = None
        if pp > 1:
            from .parallel.pp import InterleavedSchedule, PipelineSchedule
            self.schedule = (InterleavedSchedule(self.stage, g, cfg, micro_batch, chunks) if chunks > 1
                             else PipelineSchedule(self.stage, g, cfg, micro_batch))
        self._loss_acc = torch.zeros(1, dtype=torch.float32, device=device)
        self._dev_tokens = None
        self.micro_graph = MicroBatchGraph()

    def _micro_batch(self, mb, scale):
        loss = self.stage(mb[:, :-1], mb[:, 1:], scale)
        loss.backward()
        self._loss_acc += loss.detach()

    def train_step(self, tokens: torch.Tensor) -> torch.Tensor:
        """tokens: [n_seq, seq_len+1] int64 (pinned host or device). Returns the mean token loss (device scalar); with
        context parallelism every rank of the group passes the same sequences and the returned values of the group
        add up to the mean."""
        cfg = self.cfg
        n_seq = tokens.shape[0]
        assert n_seq % self.micro_batch == 0
        n_micro = n_seq // self.micro_batch
        if tokens.device != self.device:
            if self._dev_tokens is None or self._dev_tokens.shape != tokens.shape:
                self._dev_tokens = torch.empty(tokens.shape, dtype=tokens.dtype, device=self.device)
            self._dev_tokens.copy_(tokens, non_blocking=True)
            tokens = self._dev_tokens
        if self.cp_ctx is not None:
            # this rank's part of every sequence: positions [lo, lo + s) as inputs, [lo + 1, lo + s + 1) as targets
            s_local = cfg.seq_len // self.parallel.cp
            lo = self.cp_ctx.rank * s_local
            tokens = tokens[:, lo:lo + s_local + 1]
        # health: the status words copied at the end of the previous step (no synchronisation); a wait that gave
        # up inside a fused kernel means that step's gradients or parameters are not valid
        self.check_health(wait=False)
        self.stage.zero_grad_buffer()
        self._loss_acc.zero_()
        # loss is summed over tokens of this rank's micro-batches and scaled so that the sum over
        # all data-parallel ranks is the global mean
        scale = 1.0 / (n_seq * cfg.seq_len * self.parallel.dp)
        if self.schedule is not None:
            self.schedule.run(tokens, n_micro, scale, self._loss_acc)
        else:
            replay = self.micro_graph.ready(self, (self.micro_batch, tokens.shape[1]), scale)
            for i in range(n_micro):
                mb = tokens[i * self.micro_batch:(i + 1) * self.micro_batch]
                if replay:
                    self.micro_graph.run(mb)
                else:
                    self._micro_batch(mb, scale)
        self.stage.post_backward_sync_autograd_grads()
        if self.groups is not None:
            self.groups.sync_shared_grads(self.stage)
        self.opt.step(grad_scale=1.0)
        if self.expert_opt is not None:
            self.expert_opt.step(coef=self.opt._coef)
        for c in self._comms():
            c.post_status_read()
        return self._loss_acc * self.parallel.dp  # this rank's mean loss

    @torch.no_grad()
    def eval_step(self, tokens: torch.Tensor) -> torch.Tensor:
        """Mean token loss of `tokens` [n_seq, seq_len + 1] under the current parameters: forward passes only, no
        gradient, no update. Same conventions as train_step: each data-parallel rank passes its own sequences, and
        the returned values add up over the ranks that hold a loss exactly as train_step's do."""
        cfg = self.cfg
        n_seq = tokens.shape[0]
        assert n_seq % self.micro_batch == 0
        n_micro = n_seq // self.micro_batch
        if tokens.device != self.device:
            tokens = tokens.to(self.device, non_blocking=True)
        if self.cp_ctx is not None:
            s_local = cfg.seq_len // self.parallel.cp
            lo = self.cp_ctx.rank * s_local
            tokens = tokens[:, lo:lo + s_local + 1]
        acc = torch.zeros(1, dtype=torch.float32, device=self.device)
        scale = 1.0 / (n_seq * cfg.seq_len * self.parallel.dp)
        if self.schedule is not None:
            self.schedule.run_forward_only(tokens, n_micro, scale, acc)
        else:
            for i in range(n_micro):
                mb = tokens[i * self.micro_batch:(i + 1) * self.micro_batch]
                acc += self.stage(mb[:, :-1], mb[:, 1:], scale)
        return acc * self.parallel.dp

    def _comms(self):
        g = self.groups
        return [c for c in ((g.tp_comm, g.dp_comm, g.pp_comm, getattr(g, "ep_comm", None), getattr(g, "cp_comm", None))
                            if g is not None else ())
                if c is not None]

    def check_health(self, wait: bool = True) -> None:
        """Raise coccl_b200.parallel.comm.PeerLost if a bounded wait inside a fused collective, a tensor-parallel
        fusion or the expert exchange gave up during an earlier step, and RuntimeError for a GEMM pipeline error.
        `wait=True` first waits for the copies of the status words queued by the last step."""
        for c in self._comms():
            c.poll_status(wait=wait)
        if wait:
            from .ops import gemm as G
            G.check_errors()


_OWN_CODE = _own_code()
