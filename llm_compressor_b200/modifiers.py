"""``GPTQModifier`` and ``QuantizationModifier`` with the reference's fields, lifecycle hooks
and error behaviour, running on the b200q kernels.

Mirrors src/llmcompressor/modifiers/gptq/base.py:47-400,
src/llmcompressor/modifiers/quantization/quantization/{base.py:24-110,mixin.py:56-440},
src/llmcompressor/modifiers/quantization/calibration.py:36-162 and the hook helper
src/llmcompressor/modifiers/utils/hooks.py:19-110.  Only weight quantisation is on this
package's path: schemes that also name input activations keep that information for the
checkpoint format, nothing is calibrated for it.
"""
from __future__ import annotations

import collections
import contextlib
import functools
import re
import time
import warnings
from typing import Any, Iterable, Optional

import torch

from . import dist as bdist
from . import gptq, ops
from ._lib import B200QError, stream_of
from .observers import MemorylessMinMaxObserver, Observer, direct_qparams, fuse_weight_observers
from .streams import run_concurrent, run_queued
from .quant_args import (PRESET_SCHEMES, QuantizationArgs, QuantizationScheme,
                         preset_name_to_scheme)

__all__ = ["GPTQModifier", "QuantizationModifier", "match_named_modules", "HooksMixin"]

_STATIC = "static"
_UNSET = object()


# ------------------------------------------------------------------------------------------
# module matching (compressed-tensors utils/match.py:34-70,344-456)
@functools.lru_cache(maxsize=1024)
def _class_names(cls: type) -> frozenset:
    return frozenset(c.__name__ for c in cls.__mro__)


def _match_one(name: str, module: torch.nn.Module, target: str) -> bool:
    if target.startswith("re:"):
        return re.match(target[3:], name) is not None
    return name == target or target in _class_names(type(module))


def match_named_modules(model: torch.nn.Module, targets: Iterable[str], ignore: Iterable[str] = ()):
    """(name, module) pairs selected by ``targets`` and not by ``ignore``, in
    ``model.named_modules()`` order.  A target selects a module if it equals its name, if a
    ``re:`` target matches the name from its start, or if it names a class in the module's MRO."""
    targets, ignore = list(targets or []), list(ignore or [])
    out = []
    for name, module in model.named_modules():
        for t in targets:
            if _match_one(name, module, t):
                break
        else:
            continue
        for t in ignore:
            if _match_one(name, module, t):
                break
        else:
            out.append((name, module))
    return out


# ------------------------------------------------------------------------------------------
class HooksMixin:
    """Forward hooks that can be switched off globally (hooks.py:54-66)."""

    _HOOKS_DISABLED = False

    def __init__(self):
        self._hooks: list = []

    @classmethod
    @contextlib.contextmanager
    def disable_hooks(cls):
        prev = HooksMixin._HOOKS_DISABLED
        HooksMixin._HOOKS_DISABLED = True
        try:
            yield
        finally:
            HooksMixin._HOOKS_DISABLED = prev

    def register_hook(self, module: torch.nn.Module, fn, kind: str = "forward", with_kwargs: bool = False):
        def wrapped(*a, **k):
            if HooksMixin._HOOKS_DISABLED:
                return None
            return fn(*a, **k)
        register = getattr(module, f"register_{kind}_hook")
        handle = register(wrapped, with_kwargs=True) if with_kwargs else register(wrapped)
        self._hooks.append(handle)
        return handle

    def remove_hooks(self):
        for h in self._hooks:
            h.remove()
        self._hooks = []


# ------------------------------------------------------------------------------------------
class QuantizationMixin(HooksMixin):
    """Scheme resolution, qparam attachment and observer life cycle (mixin.py:56-440)."""

    def __init__(self, config_groups=None, targets="Linear", ignore=None, scheme=None,
                 kv_cache_scheme=None, weight_observer=None, input_observer=None,
                 output_observer=None, observer=None, bypass_divisibility_checks=False):
        HooksMixin.__init__(self)
        self.config_groups = config_groups
        self.targets = [targets] if isinstance(targets, str) else list(targets)
        self.ignore = list(ignore or [])
        self.scheme = scheme
        self.kv_cache_scheme = None if kv_cache_scheme is None else QuantizationArgs.of(kv_cache_scheme)
        self.weight_observer = weight_observer
        self.input_observer = input_observer
        self.output_observer = output_observer
        self.observer = observer
        self.bypass_divisibility_checks = bypass_divisibility_checks
        if self.kv_cache_scheme is not None:
            kv = self.kv_cache_scheme
            if kv.strategy != "tensor" or kv.dynamic is not False:
                raise NotImplementedError("kv-cache scales are calibrated per tensor and statically "
                                          f"(got strategy {kv.strategy!r}, dynamic {kv.dynamic!r})")
        self._resolved: Optional[dict] = None
        self._module_names: dict = {}
        self._attention_names: dict = {}   # attention modules that carry kv-cache scales

    def recipe_args(self) -> dict:
        """Constructor arguments for ``recipe.yaml`` (unset ones are left out by the writer)."""
        args = dict(config_groups=self.config_groups, targets=self.targets, ignore=self.ignore, scheme=self.scheme,
                    kv_cache_scheme=None if self.kv_cache_scheme is None else _plain_args(self.kv_cache_scheme),
                    weight_observer=self.weight_observer,
                    input_observer=self.input_observer, output_observer=self.output_observer,
                    observer=self.observer,
                    bypass_divisibility_checks=self.bypass_divisibility_checks or None)
        if isinstance(args["config_groups"], dict):
            args["config_groups"] = {k: (_plain_scheme(v)) for k, v in args["config_groups"].items()}
        return args

    # ---- scheme resolution ---------------------------------------------------------------
    def _apply_observer_overrides(self, scheme: QuantizationScheme) -> QuantizationScheme:
        has_individual = any(o is not None for o in (self.weight_observer, self.input_observer,
                                                     self.output_observer))
        if has_individual and self.observer is not None:
            raise ValueError(
                "Cannot specify both individual observer parameters (weight_observer, "
                "input_observer, output_observer) and observer dict. "
                "Please use either individual parameters or the observer dict.")
        weight_obs = self.weight_observer
        if self.observer is not None:
            weight_obs = self.observer.get("weights", weight_obs)
        if weight_obs is not None and scheme.weights is not None:
            scheme.weights = scheme.weights.model_copy(update={"observer": weight_obs})
        return scheme

    def resolve_quantization_config(self) -> dict:
        """``{"group_i": QuantizationScheme}`` (mixin.py:335-386)."""
        scheme, config_groups = self.scheme, self.config_groups
        if scheme is not None and config_groups is not None:
            raise ValueError("Please specify either `scheme` or `config_groups`")
        groups = {}
        if scheme is not None:
            if isinstance(scheme, str):
                scheme = {scheme: self.targets}
            for idx, (key, tg) in enumerate(scheme.items()):
                if key.upper() not in PRESET_SCHEMES:
                    raise ValueError(f"Unknown preset scheme {key}")
                tg = [tg] if isinstance(tg, str) else list(tg)
                groups[f"group_{idx}"] = self._apply_observer_overrides(preset_name_to_scheme(key, tg))
        elif config_groups:
            for name, g in config_groups.items():
                if isinstance(g, dict):
                    w = g.get("weights")
                    g = QuantizationScheme(targets=list(g.get("targets", self.targets)),
                                           weights=None if w is None else QuantizationArgs.of(w),
                                           input_activations=g.get("input_activations"))
                elif not isinstance(g, QuantizationScheme):
                    g = QuantizationScheme(targets=list(g.targets),
                                           weights=None if g.weights is None else QuantizationArgs.of(g.weights),
                                           input_activations=getattr(g, "input_activations", None))
                groups[name] = self._apply_observer_overrides(g)
        else:
            groups["group_0"] = self._apply_observer_overrides(
                QuantizationScheme(targets=list(self.targets), weights=QuantizationArgs(num_bits=8)))
        return groups

    # ---- attach / detach -------------------------------------------------------------------
    def initialize_quantization(self, model: torch.nn.Module) -> None:
        """Attach ``quantization_scheme`` and empty scale / zero-point (/ global scale / g_idx)
        parameters to every targeted module (CT lifecycle/initialize.py:132-254)."""
        groups = self.resolve_quantization_config()
        self._resolved = groups
        bad, zero_points = [], {}
        for scheme in groups.values():
            for name, module in match_named_modules(model, scheme.targets, self.ignore):
                weight = getattr(module, "weight", None)
                if weight is None or weight.ndim != 2:
                    continue
                if isinstance(module, torch.nn.Embedding):
                    continue
                w = scheme.weights
                if w is None:
                    continue
                N, K = weight.shape
                if (w.strategy in ("group", "tensor_group") and K >= w.group_size and K % w.group_size
                        and not self.bypass_divisibility_checks):
                    bad.append((name, K, w.group_size))
                    continue
                _set_plain(module, "quantization_scheme", scheme)
                _set_plain(module, "quantization_status", "initialized")   # "frozen" once its qparams are written
                self._module_names[module] = name
                dev, dt = weight.device, weight.dtype
                shape = w.qparam_shape(N, K)

                def reg(pname, t):
                    module.register_parameter(pname, torch.nn.Parameter(t, requires_grad=False))
                if w.strategy == "tensor_group":
                    reg("weight_global_scale", torch.empty(1, dtype=torch.float32, device=dev))
                reg("weight_scale", torch.empty(shape, dtype=dt if dt.is_floating_point else torch.float16,
                                                device=dev))
                zero_point = torch.empty(shape, dtype=w.zp_dtype, device=dev)
                reg("weight_zero_point", zero_point)
                zero_points.setdefault(dev, []).append(zero_point)
                if w.actorder == "group":
                    reg("weight_g_idx", torch.full((K,), -1, dtype=torch.int32, device=dev))
                a = scheme.input_activations
                if a is not None and a.dynamic is not True:
                    # statically calibrated input activations (CT lifecycle/initialize.py:164-254):
                    # a per-tensor scale / zero point, or (dynamic "local") only the global scale
                    if a.strategy == "tensor_group":
                        reg("input_global_scale", torch.empty(1, dtype=torch.float32, device=dev))
                    if a.dynamic is False:
                        if a.strategy != "tensor":
                            raise NotImplementedError("static input activations are supported per tensor")
                        reg("input_scale", torch.empty(1, dtype=dt if dt.is_floating_point else torch.float16,
                                                       device=dev))
                        reg("input_zero_point", torch.zeros(1, dtype=a.zp_dtype, device=dev))
        for tensors in zero_points.values():
            # one launch clears them all (a launch each: 8 us of host time); for one a plain memset, 3 us less on the device
            if len(tensors) == 1:
                tensors[0].view(torch.int8).zero_()
            else:
                torch._foreach_zero_([t.view(torch.int8) for t in tensors])
        if self.kv_cache_scheme is not None:
            # attention modules get k_scale / v_scale (CT lifecycle/initialize.py:255-310); the scheme
            # sits on the module as its input_activations, as the reference's config resolution puts it
            kv = self.kv_cache_scheme
            attn = match_named_modules(model, KV_CACHE_TARGETS, self.ignore)
            if not attn:
                raise ValueError(f"kv_cache_scheme given but no module matches {KV_CACHE_TARGETS}")
            for name, module in attn:
                first = next(module.parameters(), None)
                if first is None:
                    raise ValueError(f"attention module {name} has no parameters to take device and dtype from")
                module.quantization_scheme = QuantizationScheme(targets=list(KV_CACHE_TARGETS), weights=None,
                                                                input_activations=kv)
                module.quantization_status = "initialized"
                self._attention_names[module] = name
                dt = first.dtype if first.dtype.is_floating_point else torch.float16
                for base in ("k", "v"):
                    module.register_parameter(f"{base}_scale", torch.nn.Parameter(
                        torch.empty(1, dtype=dt, device=first.device), requires_grad=False))
                    if not kv.symmetric:
                        module.register_parameter(f"{base}_zero_point", torch.nn.Parameter(
                            torch.zeros(1, dtype=kv.zp_dtype, device=first.device), requires_grad=False))
        if bad:
            lines = "\n".join(f"  {n}: columns {k} not divisible by group_size {g}" for n, k, g in bad)
            raise ValueError(
                "The following layers have weight column counts that are not divisible by the "
                f"quantization group size:\n{lines}\nAdd them to `ignore` or set "
                "bypass_divisibility_checks=True")

    def quantized_modules(self, model: torch.nn.Module):
        return [(n, m) for n, m in model.named_modules() if m in self._module_names and hasattr(m, "quantization_scheme")]

    def start_calibration(self, model: torch.nn.Module) -> None:
        shared = False   # some weights have a global scale that siblings share
        for _, module in self.quantized_modules(model):
            w = module.quantization_scheme.weights
            _set_plain(module, "weight_observer", Observer.load_from_registry(
                w.observer or "memoryless_minmax", base_name="weight", args=w))
            shared = shared or w.strategy == "tensor_group"
            a = module.quantization_scheme.input_activations
            if a is not None and a.dynamic is not True:
                name = a.observer if a.observer not in (None, "memoryless_minmax") else "minmax"
                module.input_observer = Observer.load_from_registry(name, base_name="input", args=a)
                self.register_hook(module, _calibrate_input_hook, "forward_pre")
        for module in self._attention_names:
            a = module.quantization_scheme.input_activations
            name = a.observer if a.observer not in (None, "memoryless_minmax") else "minmax"
            module.k_observer = Observer.load_from_registry(name, base_name="k", args=a)
            module.v_observer = Observer.load_from_registry(name, base_name="v", args=a)
            self.register_hook(module, _observing_cache_hook, "forward_pre", with_kwargs=True)
        if shared:
            fuse_weight_observers(model)

    @property
    def calibrates_activations(self) -> bool:
        """True when some resolved scheme has statically calibrated input activations."""
        groups = self._resolved if self._resolved is not None else self.resolve_quantization_config()
        return self.kv_cache_scheme is not None or any(
            s.input_activations is not None and s.input_activations.dynamic is not True for s in groups.values())

    def update_activation_qparams(self, modules) -> None:
        """Epoch end for activation observers: combine the ranks' statistics, then write
        ``input_scale`` / ``input_zero_point`` / ``input_global_scale``
        (quantization/base.py:83-108, calibration.py:109-162)."""
        modules = list(modules)
        pending = []
        seen = []
        for base in ("input", "k", "v"):
            mods = [m for m in modules if getattr(m, f"{base}_observer", None) is not None
                    and getattr(m, f"{base}_observer").has_statistics]
            if mods and bdist.is_distributed():
                for m in mods:
                    pending.extend(getattr(m, f"{base}_observer").sync_activation_stats())
            seen.append((base, mods))
        bdist.wait_for_comms(pending)
        for base, mods in seen:
            update_qparams(mods, base)
            if base == "v":
                for m in mods:
                    m.quantization_status = "frozen"

    def end_calibration(self, model: torch.nn.Module) -> None:
        self.remove_hooks()
        for module in list(self._module_names) + list(self._attention_names):
            for name in ("weight_observer", "input_observer", "k_observer", "v_observer"):
                module.__dict__.pop(name, None)


KV_CACHE_TARGETS = ("re:.*self_attn$",)   # the reference's match for attention modules (mixin.py:216-218)


class _ObservingCache:
    """Stands in for ``past_key_values`` during a calibration forward of an attention module: the
    attention calls ``update(key_states, value_states, layer_idx, ...)`` with the post-rotary keys
    and the values, [batch, kv_heads, tokens, head_dim], which are what a cache would store.  They
    go to the module's k / v observers and on to the cache that was passed in, if any
    (compressed-tensors modeling/kvcache.py:29-84, calibration.py:187-196)."""

    def __init__(self, module, inner):
        self.module, self.inner = module, inner

    def update(self, key_states, value_states, *args, **kwargs):
        self.module.k_observer(key_states)
        self.module.v_observer(value_states)
        if self.inner is not None:
            return self.inner.update(key_states, value_states, *args, **kwargs)
        return key_states, value_states

    def __getattr__(self, name):   # anything else an attention implementation asks of a cache
        inner = self.__dict__.get("inner")
        if inner is None:
            raise AttributeError(name)
        return getattr(inner, name)


def _observing_cache_hook(module, args, kwargs):
    import inspect
    name = "past_key_values" if "past_key_values" in inspect.signature(module.forward).parameters \
        else "past_key_value"
    kwargs[name] = _ObservingCache(module, kwargs.get(name))
    return args, kwargs


def _calibrate_input_hook(module, args):
    """calibration.py:165-170: the input observer sees every calibration batch."""
    module.input_observer(args[0] if isinstance(args, tuple) else args)


def observe(modules: Iterable[torch.nn.Module], base_name: str = "weight") -> None:
    for m in modules:
        obs = getattr(m, f"{base_name}_observer", None)
        if obs is not None:
            obs(m.weight.data)


def update_qparams(modules: Iterable[torch.nn.Module], base_name: str = "weight") -> None:
    """Copy the observer's scale / zero point / global scale into the module's parameters
    (calibration.py:109-162)."""
    for m in modules:
        obs = getattr(m, f"{base_name}_observer", None)
        if obs is None:
            continue
        if not obs.has_statistics:
            warnings.warn(f"Observer of {type(m).__name__} has no statistics; qparams not updated")
            continue
        qp = obs.get_qparams()
        _write_qparams(m, base_name, qp["scale"], qp["zero_point"], qp["global_scale"])


def _write_qparams(m, base_name, scale, zero_point, global_scale) -> None:
    # (the scale is absent for locally dynamic activations, which have a global scale only; symmetric kv-cache scales
    # carry no zero point)
    params = m._parameters
    written = [("scale", scale)]
    if params.get(base_name + "_scale") is not None:
        written.append(("zero_point", zero_point))
    if global_scale is not None:
        written.append(("global_scale", global_scale))
    for what, val in written:
        p = params.get(f"{base_name}_{what}")
        if p is not None:
            _put(p, val)
    if base_name == "weight":
        _set_plain(m, "quantization_status", "frozen")


def _write_shared_qparams(modules):
    """Parameters of the weights that share a global scale (and of single ones with a global scale), all of a group in two
    launches; returns the modules that are left."""
    by_observer = {id(m.weight_observer): m for m in modules if m.weight_observer.args.strategy == "tensor_group"}
    if not by_observer:
        return modules
    done = set()
    for m in modules:
        obs = m.weight_observer
        if id(obs) not in by_observer or id(m) in done:
            continue
        observers = [obs] + obs._fused
        group = [by_observer.get(id(o)) for o in observers]
        if any(g is None or type(o) is not MemorylessMinMaxObserver or o.has_statistics or o.args != obs.args
               for o, g in zip(observers, group)):
            continue
        into = [[g._parameters.get("weight_" + name) for g in group] for name in ("scale", "zero_point", "global_scale")]
        if any(p is None for ps in into for p in ps):
            continue
        if ops.shared_qparams([g.weight.data for g in group], obs.args, *[[p.data for p in ps] for ps in into]):
            for g in group:
                done.add(id(g))
                _set_plain(g, "quantization_status", "frozen")
    return [m for m in modules if id(m) not in done]


def _set_plain(module, name, value) -> None:
    """``setattr`` for a value that is no parameter, buffer or submodule: torch's own looks for all of these first, in
    Python, at 4 us an attribute."""
    object.__setattr__(module, name, value)


def _put(p: torch.Tensor, val: torch.Tensor) -> None:
    """Give parameter ``p`` the values of ``val``, a fresh tensor nobody else writes: no copy where it can stand in."""
    if val.shape != p.shape:
        val = val.reshape(p.shape)
    if val.dtype == p.dtype and val.device == p.device and val.is_contiguous():
        p.data = val
    else:
        p.data.copy_(val)


# ------------------------------------------------------------------------------------------
class QuantizationModifier(QuantizationMixin):
    """Round-to-nearest weight quantisation: observe weights, write qparams; the weight is
    left as is until it is packed at save time (quantization/base.py:24-110)."""

    @property
    def requires_calibration_data(self) -> bool:
        return self.calibrates_activations

    def on_initialize(self, model, **_):
        self.initialize_quantization(model)
        return True

    def on_calibration_start(self, model, **_):
        self.start_calibration(model)

    def on_sequential_epoch_end(self, model, modules: Iterable[torch.nn.Module], **_):
        modules = list(modules)
        if self.calibrates_activations:
            self.update_activation_qparams(modules)
        modules = [m for m in modules if "weight_observer" in m.__dict__
                   and getattr(m, "quantization_status", None) != "frozen"]
        if bdist.is_distributed():
            # owners by weight size; each rank observes its share, scales are broadcast
            items, rank_to, to_rank = bdist.greedy_bin_packing(
                list(modules), bdist.world_size(), item_weight_fn=lambda m: m.weight.numel())
            mine = rank_to[bdist.rank()]
            observe(mine)
            update_qparams(mine)
            bdist.broadcast_module_params(items, to_rank,
                                          ("weight_scale", "weight_zero_point", "weight_global_scale"))
            for m in items:
                m.quantization_status = "frozen"
        else:
            # most weights: statistics and parameters in one launch
            rest = []
            modules = _write_shared_qparams(modules)
            for m in modules:
                params = m._parameters
                scale, zp = params.get("weight_scale"), params.get("weight_zero_point")
                into = None if scale is None or zp is None else (scale.data, zp.data)
                if into is not None and direct_qparams([m.weight_observer], [m.weight.data], into) is not None:
                    _set_plain(m, "quantization_status", "frozen")
                else:
                    rest.append(m)
            if rest:
                observe(rest)
                update_qparams(rest)

    def pending_modules(self):
        """Targeted modules whose parameters have not been written yet (modules behind the
        sequential blocks)."""
        return [m for m in self._module_names if hasattr(m, "weight_observer")
                and getattr(m, "quantization_status", None) != "frozen"]

    def on_calibration_end(self, model, **_):
        self.end_calibration(model)

    def on_finalize(self, model, **_):
        return True


class GPTQModifier(QuantizationMixin):
    """GPTQ weight quantisation (gptq/base.py:47-400).

    Forward hooks accumulate H += 2 X^T X per calibration batch; at the end of each sequential
    epoch the modules of that epoch are observed and quantised column block by column block.
    Modules that receive the very same input tensor (q/k/v, gate/up, experts under all-expert
    calibration) share one Hessian accumulation and one factorisation; set
    ``share_hessians=False`` to keep one per module like the reference.  The solves of different
    Hessians run concurrently on up to ``parallel_streams`` CUDA streams (1: one after another
    on the current stream, like the reference).  Calibration batches smaller than
    ``hessian_stage_tokens`` (and than ``_DIRECT_TOKENS``) tokens are gathered and added to the Hessian together (0: one kernel
    call per batch).  When an epoch holds ``batch_small_hessians`` or more Hessians of one width of
    at most ``small_hessian_columns`` columns (the experts of a mixture-of-experts layer), their
    factorisations and sweeps run as batched launches that serve all of them, instead of
    dozens of launches per module (0 switches this off).
    """

    requires_calibration_data = True

    def __init__(self, block_size: int = 128, dampening_frac: Optional[float] = 0.01,
                 actorder: Any = _UNSET, offload_hessians: bool = False, share_hessians: bool = True,
                 parallel_streams: int = 4, hessian_stage_tokens: int = 32768,
                 batch_small_hessians: int = 16, small_hessian_columns: int = 2048, **quant_kwargs):
        kw = dict(quant_kwargs)
        kw.setdefault("targets", "Linear")
        super().__init__(**kw)
        self.block_size = block_size
        self.dampening_frac = dampening_frac
        self.actorder = actorder
        self.offload_hessians = offload_hessians
        self.share_hessians = share_hessians
        self.parallel_streams = parallel_streams
        self.hessian_stage_tokens = hessian_stage_tokens
        self.batch_small_hessians = batch_small_hessians
        self.small_hessian_columns = small_hessian_columns
        self._groups: dict = {}        # module -> _HessianGroup
        self._by_input: dict = {}      # _input_key of a batch of this epoch -> the group that took it last
        self._num_samples: dict = {}   # module -> None (membership: modules awaiting compression)
        self.trace = None              # optional callback(event: str, module | None) for instrumentation
        self._hooked: list = []        # every module that got a calibration hook
        self._done: set = set()        # modules whose quantised weight has been written
        self.losses: dict = {}

    def recipe_args(self) -> dict:
        args = super().recipe_args()
        args.update(block_size=self.block_size, dampening_frac=self.dampening_frac,
                    offload_hessians=self.offload_hessians or None)
        if self.actorder is not _UNSET:
            args["actorder"] = self.actorder   # None is dropped by the writer, as the reference drops it
        return args

    # ---- config ------------------------------------------------------------------------------
    def resolve_quantization_config(self) -> dict:
        groups = super().resolve_quantization_config()

        def resolve(existing):
            if self.actorder is _UNSET:  # sentinel default only fills an unset scheme value
                return "weight" if existing is None else existing
            mine = QuantizationArgs(num_bits=4, group_size=128, actorder=self.actorder).actorder \
                if self.actorder not in (None, False) else None
            if existing is None or mine == existing:
                return mine
            raise ValueError(
                "Cannot resolve activation ordering when both `GPTQModifier.actorder` and "
                f"`QuantizationScheme.actorder` are provided and differ ({self.actorder}, {existing}). "
                "Either unset `GPTQModifier.actorder` or remove `actorder` from config groups.")

        for scheme in groups.values():
            w = scheme.weights
            if w is None:
                continue
            # the modifier-level setting is applied to every strategy, as the reference does by
            # assigning past the argument validation (base.py:176-192): "weight"/"static" then
            # permutes the sweep of channel / tensor / block schemes too
            a = resolve(w.actorder)
            if a == "group" and w.strategy not in ("group", "tensor_group"):
                warnings.warn(f"ActivationOrdering.GROUP is not compatible with strategy={w.strategy}; "
                              "falling back to actorder=None for this scheme.")
                a = None
            scheme.weights = _with_actorder(w, a)
        return groups

    # ---- lifecycle -----------------------------------------------------------------------------
    def on_initialize(self, model, **_):
        self.initialize_quantization(model)
        return True

    def on_calibration_start(self, model, **_):
        self.start_calibration(model)
        self._hooked, self._done = [], set()   # a fresh calibration
        added = False
        for _, module in self.quantized_modules(model):
            if isinstance(module, torch.nn.Embedding):
                continue
            if getattr(module, "quantization_scheme", None) is None or module.quantization_scheme.weights is None:
                continue
            self.register_hook(module, self.calibrate_module, "forward")
            self._hooked.append(module)
            added = True
        if not added:
            raise ValueError(
                "GPTQModifier requires a weight quantization config be specified by this modifier or a "
                "modifier preceding it")

    def pending_modules(self):
        """Hooked modules that have not been compressed yet."""
        return [m for m in self._hooked if m not in self._done]

    def calibrate_module(self, module, args, _output):
        if module in self._done:
            return
        inp = args[0]
        group = self._groups.get(module)
        if group is None:
            group = self._find_shared(inp) if self.share_hessians else None
            if group is not None:
                group.members.append(module)
                self._groups[module] = group
                self._num_samples[module] = None
                return   # the batch is in the Hessian already
            else:
                group = _HessianGroup(module, offload=self.offload_hessians, stage_tokens=self.hessian_stage_tokens)
            self._groups[module] = group
            self._num_samples[module] = None
        elif group.same_input(inp):
            return
        elif module is not group.members[0]:
            # membership was decided on the first batch; the first member adds every batch and
            # the others must keep receiving that very tensor
            raise RuntimeError(
                f"{self._module_names.get(module, type(module).__name__)} shared a Hessian with "
                f"{self._module_names.get(group.members[0], type(group.members[0]).__name__)} because both received "
                "the same input on the first calibration batch, but its input differs on a later batch; "
                "set GPTQModifier(share_hessians=False)")
        group.accumulate(inp)
        self._by_input[_input_key(inp)] = group

    def _find_shared(self, inp):
        # by address first: an epoch of 64 experts has 65 groups to look through for each new module
        g = self._by_input.get(_input_key(inp))
        if g is None:
            return None
        if g.same_input(inp):
            return g
        for g in {id(g): g for g in self._groups.values()}.values():
            if g.same_input(inp):
                return g
        return None

    def on_sequential_epoch_end(self, model, modules: Iterable[torch.nn.Module], **_):
        modules = list(modules)
        if self.calibrates_activations:
            self.update_activation_qparams(modules)
        mods = [m for m in modules if m in self._num_samples]
        # the weight observers are called by the solves themselves (gptq._sweep_input), on the rank
        # and stream that quantises the module, next to the rest of its work
        self.compress_modules(mods)

    def _trace(self, event, module=None):
        if self.trace is not None:
            self.trace(event, module)

    def compress_modules(self, modules=None):
        modules = list(self._num_samples.keys()) if modules is None else list(modules)
        self._by_input.clear()
        if not bdist.is_distributed():
            self._trace("solve")
            self.compress_module_list(modules)
            self._trace("done")
            return
        # owners by Hessian width over the distinct Hessians (base.py:306-318).  A Hessian shared by
        # many modules (the gate / up projections of every expert under all-expert calibration)
        # would make its owner sweep all of them alone: such a Hessian is summed onto every rank
        # instead, every rank factors it, and its modules are dealt out round robin.
        world = bdist.world_size()
        groups = list({id(self._groups[m]): self._groups[m] for m in modules}.values())
        members = {id(g): [m for m in modules if self._groups[m] is g] for g in groups}
        spread = [g for g in groups if len(members[id(g)]) >= 2 * world]
        owned = [g for g in groups if len(members[id(g)]) < 2 * world]
        items, rank_to, to_rank = bdist.greedy_bin_packing(owned, world, item_weight_fn=lambda g: g.H.shape[0])
        for g in spread:
            to_rank[g] = None
        items = items + spread
        for g in items:
            g.flush()   # staged calibration tokens
        self._trace("reduce")
        bdist.reduce_hessians(items, to_rank)
        mod_rank = {}    # before the solve drops the groups
        for g in items:
            for i, m in enumerate(members[id(g)]):
                mod_rank[m] = to_rank[g] if to_rank[g] is not None else i % world
        mine = [m for m in modules if mod_rank[m] == bdist.rank()]
        self._trace("solve")
        self.compress_module_list(mine)
        self._trace("broadcast")
        bdist.broadcast_module_params(modules, mod_rank, ("weight", "weight_scale", "weight_zero_point",
                                                          "weight_g_idx", "weight_global_scale"))
        for m in modules:
            self._num_samples.pop(m, None)
            self._groups.pop(m, None)
            m.quantization_status = "frozen"
            self._done.add(m)
        self._trace("done")

    def compress_module_list(self, module_list):
        """Quantise the modules; the modules of one Hessian form a job (one factorisation per
        act-order setting, then their sweeps) and jobs run concurrently on side streams."""
        by_group: dict = {}
        for module in module_list:
            by_group.setdefault(id(self._groups[module]), []).append(module)
        jobs = sorted(by_group.values(), key=lambda mods: -mods[0].weight.shape[1])
        if not jobs:
            return
        device = jobs[0][0].weight.device
        if self.batch_small_hessians and self.block_size == 128:
            # small problems that come in numbers: many Hessians of one width, or one Hessian
            # shared by many modules (the gate / up projections under all-expert calibration)
            width = collections.Counter()
            for mods in jobs:
                width[mods[0].weight.shape[1]] += len(mods)
            small = [mods for mods in jobs if mods[0].weight.shape[1] <= self.small_hessian_columns
                     and width[mods[0].weight.shape[1]] >= self.batch_small_hessians]
            if small:
                taken = {id(mods) for mods in small}
                jobs = [mods for mods in jobs if id(mods) not in taken]
                self._compress_small_jobs(small)
        if jobs:
            if len(jobs) <= self.parallel_streams:
                run_queued([lambda mods=mods: self._queue_group(mods) for mods in jobs], device)
            else:
                run_concurrent([lambda mods=mods: self._compress_group(mods) for mods in jobs], device,
                               max_streams=self.parallel_streams)
            for mods in _loss_order(jobs):
                for m in mods:
                    name = self._module_names.get(m, type(m).__name__)
                    if name in self.losses:
                        self.losses[name] = self.losses.pop(name)

    def _queue_factors(self, module_list, make_factor):
        """Take the modules of one Hessian out of the pending tables and give each the factor of its
        act-order setting, made by ``make_factor(H, actorder)`` once per distinct setting.
        Returns ([(module, qargs, factor)], the Hessian's device status word or None)."""
        factors = {}
        left = {module.quantization_scheme.weights.actorder for module in module_list}
        taken, status = [], None
        for module in module_list:
            group = self._groups.pop(module)
            self._num_samples.pop(module, None)
            qargs = module.quantization_scheme.weights
            if qargs.actorder not in factors:
                left.discard(qargs.actorder)
                H = group.finalized(keep=bool(left))  # the factorisation consumes its argument
                factors[qargs.actorder] = make_factor(H, qargs.actorder)
                self._trace("job_factored", module)
            status = group.status   # (after the sum has been handed over)
            taken.append((module, qargs, factors[qargs.actorder]))
        return taken, status

    @staticmethod
    def _check_status_words(words):
        words = [w for w in words if w is not None]
        if words and int(torch.cat([w.reshape(-1)[:1] for w in words]).abs().amax().item()) != 0:
            raise B200QError("a bounded wait inside the Hessian or GEMM kernels of this job expired; "
                             "its results are incomplete")

    def _finish_queued(self, queued, t0, batch=(), gathered=None):
        """``queued``: [(module, qargs, factor, loss, out)] of deferred solves whose factors have been
        resolved; ``batch``: those of them whose values are slices of a batch's buffers, and ``gathered``
        what ``_gather_copies`` makes of them all.  Redo the modules whose Hessian was not positive definite with the
        identity, as the reference falls back (gptq_quantize.py:157-164), then write every result to its module."""
        redo = [q for q in queued if not q[2].ok]
        # the deferred call consumed the observers' statistics: observe again before the
        # round-to-nearest redo (act-order "group" re-observes the permuted weight itself)
        for module, qargs, *_ in redo:
            if qargs.actorder != "group":
                module.weight_observer.delete_statistics(check_fused=False)
        for module, qargs, *_ in redo:
            if qargs.actorder != "group":
                module.weight_observer(module.weight.data)
        results = []
        for module, qargs, factor, loss, out in queued:
            if not factor.ok:
                with torch.no_grad():
                    loss, out = gptq.quantize_weight(module, qargs, None, blocksize=self.block_size,
                                                     percdamp=self.dampening_frac, factor=factor)
            results.append((module, loss, out))
        # one read for all the losses that are still on the device
        on_device = [i for i, (_, loss, _) in enumerate(results) if isinstance(loss, torch.Tensor)]
        if on_device:
            values = torch.stack([results[i][1].reshape(()) for i in on_device]).tolist()
            for i, v in zip(on_device, values):
                results[i] = (results[i][0], v, results[i][2])
        # the weights go back in one multi-tensor copy
        if results:
            torch._foreach_copy_([module.weight.data for module, _, _ in results],
                                 [out["weight"] for _, _, out in results])
        sliced = {id(q[0]) for q in batch if q[2].ok}
        for module, loss, out in results:
            loss = float(loss)
            name = self._module_names.get(module, type(module).__name__)
            self.losses[name] = loss
            self._log_metric(name, time.perf_counter() - t0, loss)
            if id(module) not in sliced:
                for attr, val in out.items():
                    if attr == "weight":
                        continue
                    p = getattr(module, attr, None)
                    if p is not None:
                        _put(p, val)
                    else:
                        module.register_parameter(attr, torch.nn.Parameter(val, requires_grad=False))
            _set_plain(module, "quantization_status", "frozen")
            self._done.add(module)
        if redo and batch:
            gathered = _gather_copies([(q[0], q[4]) for q in batch if q[2].ok])
        if gathered:
            copies, unset = gathered
            for module, attr, p in unset:
                module.register_parameter(attr, p)
            for into, values in copies.values():
                torch._foreach_copy_(into, values)

    def _compress_group(self, module_list):
        """Factor and sweep the modules of one Hessian."""
        self._queue_group(module_list)()

    def _queue_group(self, module_list):
        """The work of ``_compress_group`` without its end, which comes back as a callable.  Everything is
        queued on the current stream without waiting for the device; the factorisation status and the
        losses are read once at the end."""
        t0 = time.perf_counter()
        self._trace("job_start", module_list[0])
        taken, hess_status = self._queue_factors(
            module_list, lambda H, actorder: gptq.factor_for_modules(H, module_list, self.dampening_frac, actorder))
        queued = []
        for module, qargs, factor in taken:
            with torch.no_grad():
                loss, out = gptq.quantize_weight(module, qargs, None, blocksize=self.block_size,
                                                 percdamp=self.dampening_frac, factor=factor, defer=True)
            queued.append((module, qargs, factor, loss, out))
        self._trace("job_swept", module_list[0])

        def finish():
            # one read for every device status word of the job (the first wait for the device)
            self._check_status_words([out.pop("_status", None) for *_, out in queued] + [hess_status])
            gptq.resolve_factors([q[2] for q in queued])
            self._finish_queued(queued, t0)
        return finish

    def _compress_small_jobs(self, jobs):
        """Many Hessians of few columns: the same steps as ``_compress_group`` for every job, but the
        factorisations of one width and the sweeps of one weight shape and scheme are gathered
        into batched launches on the current stream."""
        t0 = time.perf_counter()
        self._trace("job_start", jobs[0][0])
        requests = []   # (H, actorder, holder): the holder receives the factor once it exists

        def ask(H, actorder):
            holder = []
            requests.append((H, actorder, holder))
            return holder

        taken, words = [], []
        _finalize_groups([self._groups[mods[0]] for mods in jobs])
        for mods in jobs:
            part, status = self._queue_factors(mods, ask)
            taken += part
            words.append(status)
        by_kind: dict = {}
        for H, actorder, holder in requests:
            by_kind.setdefault((H.shape[0], H.stride(0), actorder), []).append((H, holder))
        for (_, _, actorder), items in by_kind.items():
            if len(items) >= self.batch_small_hessians:
                factors = gptq.factor_hessians_batched([H for H, _ in items], self.dampening_frac, actorder)
            else:   # a few matrices: the tensor-core factorisation, one after another
                factors = [gptq.factor_hessian(H, self.dampening_frac, actorder, defer=True) for H, _ in items]
            for (_, holder), factor in zip(items, factors):
                holder.append(factor)
        del requests, by_kind
        by_shape, schemes = {}, {}
        for module, qargs, holder in taken:
            if id(qargs) not in schemes:
                schemes[id(qargs)] = repr(qargs)
            key = (tuple(module.weight.shape), module.weight.dtype, schemes[id(qargs)])
            by_shape.setdefault(key, []).append((module, qargs, holder[0]))
        queued, batch = [], []
        # the class with the most device work first: its sweep runs while the host prepares the others
        classes = sorted(by_shape.values(), key=lambda it: -len(it) * it[0][0].weight.shape[0]
                         * it[0][0].weight.shape[1] ** 2)
        for items in classes:
            with torch.no_grad():
                if len(items) >= 4:
                    done = gptq.quantize_weights_batched([m for m, _, _ in items], items[0][1],
                                                         [f for _, _, f in items], blocksize=self.block_size,
                                                         percdamp=self.dampening_frac)
                else:
                    done = [gptq.quantize_weight(m, q, None, blocksize=self.block_size, percdamp=self.dampening_frac,
                                                 factor=f, defer=True) for m, q, f in items]
                words += [out.pop("_status", None) for _, out in done]
            queued += [(m, q, f, loss, out) for (m, q, f), (loss, out) in zip(items, done)]
            if len(items) >= 4:
                batch += queued[-len(items):]
        self._trace("job_swept", jobs[0][0])
        gathered = _gather_copies([(q[0], q[4]) for q in batch])   # (while the device is at work)
        self._check_status_words(words)
        gptq.resolve_factors([q[2] for q in queued])
        self._finish_queued(queued, t0, batch, gathered)

    @staticmethod
    def _log_metric(name, seconds, loss):
        # shape of the reference's METRIC lines (src/llmcompressor/utils/metric_logging.py:42-65)
        import logging
        logging.getLogger("llm_compressor_b200").info("METRIC - %s time %.2fs error %.2f", name, seconds, loss)

    def on_calibration_end(self, model, **_):
        self.end_calibration(model)

    def on_finalize(self, model, **_):
        if len(self._num_samples) > 0:
            raise ValueError(f"Failed to compress {len(self._num_samples)} modules")
        missed = self.pending_modules()
        if missed:
            names = ", ".join(self._module_names.get(m, type(m).__name__) for m in missed[:8])
            raise ValueError(f"{len(missed)} targeted modules never received calibration data and were not "
                             f"compressed: {names}{' ...' if len(missed) > 8 else ''}")
        self._groups, self._num_samples, self._hooked = {}, {}, []
        return True


def _loss_order(jobs) -> list:
    """The order in which the losses of one ``compress_module_list`` call stand in ``losses``, whichever job ended first:
    by the columns of a job's chain (one for the factor, one for each sweep), or, if some Hessian has fewer than 1024
    columns, by its number of modules; then by width.  The order means nothing, and callers should look losses up by name;
    it is fixed so that callers that go through ``losses.values()`` meet the same places on every run."""
    narrow = min(mods[0].weight.shape[1] for mods in jobs) < 1024

    def length(mods):
        width = mods[0].weight.shape[1]
        return (len(mods) if narrow else width * (1 + len(mods)), width)

    return sorted(jobs, key=length)


def _gather_copies(solved):
    """{(types, device): ([parameters], [values])} of [(module, out)] whose values are slices of buffers that many modules share, for
    one copy a type, and the parameters [(module, name, parameter)] that the modules do not have yet: they get them with
    their values, no sooner (a solve that fails leaves its modules as they were).  Put in as they are, the slices would keep
    the buffer alive, and saving one module would write all of it."""
    copies: dict = {}
    unset = []
    for module, out in solved:
        params = module._parameters
        for attr, val in out.items():
            if attr == "weight":
                continue
            p = params.get(attr)   # (nearly always; a buffer or plain tensor of that name is written as well)
            if p is None:
                p = getattr(module, attr, None)
            if p is None:
                p = torch.nn.Parameter(torch.empty_like(val, memory_format=torch.contiguous_format), requires_grad=False)
                unset.append((module, attr, p))
            p = p.data
            if val.shape != p.shape:
                val = val.reshape(p.shape)
            if val.dtype.itemsize == 1 and p.dtype == val.dtype:   # (the one-launch copy takes no float8)
                p, val = p.view(torch.uint8), val.view(torch.uint8)
            into, values = copies.setdefault((p.dtype, val.dtype, p.device), ([], []))
            into.append(p)
            values.append(val)
    return copies, unset


def _plain_args(a: QuantizationArgs) -> dict:
    """QuantizationArgs as plain recipe / config values."""
    out = {}
    for k, v in vars(a).items():
        if v is None or (k == "observer_kwargs" and not v):
            continue
        out[k] = str(v).replace("torch.", "") if isinstance(v, torch.dtype) else v
    return out


def _plain_scheme(g):
    """A config group as plain data for the recipe file."""
    if isinstance(g, dict):
        return {k: (_plain_scheme(v) if isinstance(v, (dict, QuantizationArgs, QuantizationScheme)) else v)
                for k, v in g.items()}
    out = {}
    for k, v in vars(g).items():
        if v is None or v == {} or v is False:
            continue
        if isinstance(v, (QuantizationArgs, QuantizationScheme)):
            v = _plain_scheme(v)
        elif isinstance(v, torch.dtype):
            v = str(v)
        out[k] = v
    return out


def _with_actorder(qargs: QuantizationArgs, actorder):
    a = qargs.model_copy()
    object.__setattr__(a, "actorder", actorder)
    return a


def _input_key(inp: torch.Tensor):
    return inp.data_ptr(), inp.shape, inp.dtype


# Batches of this many tokens go to the Hessian as they are: the update is bound by its MMAs from about there on, and the
# copy into the staging buffer costs what the larger calls save.  Microseconds a batch, direct / staged:
#   columns        256       1024      2048      4096      5632       8192       14336
#   2048 tokens  10 / 8    11 / 8    14 / 13   34 / 34   67 / 59   136 / 115   433 / 365
#   4096         10 / 9    11 / 11   19 / 21   56 / 65  112 / 116  248 / 229   759 / 748
#   8192         10 / 10   15 / 17   31 / 39  108 / 127 199 / 250  526 / 531  1524 / 1542
# One line for all widths is within 8 % of the better side at 4096 tokens, 15 % (1.5 us) below 512 columns.
_DIRECT_TOKENS = 4096


class _HessianGroup:
    """One Hessian shared by the modules that see the same input.

    Small calibration batches (below ``stage_tokens`` and ``_DIRECT_TOKENS``) are gathered in a bf16
    staging buffer and added with one kernel call per ``stage_tokens`` tokens: the symmetric rank-k
    update re-reads and re-writes the lower triangle of H on every call."""

    def __init__(self, module, offload=False, stage_tokens: int = 0):
        self.members = [module]
        K = module.weight.shape[1]
        self.device = module.weight.device
        self._home = self._stage_home = self._stream()   # that sum and staging buffer were allocated on
        # one allocation (and one launch to clear it) for the sum and the word that a bounded wait running out sets
        both = torch.zeros(K * K + 1, dtype=torch.float32, device=self.device)
        self.H = both[:K * K].view(K, K)
        self.n = 0
        self._last = None  # (tensor kept alive, version) of the batch accumulated last
        self.status = both[K * K:].view(torch.int32)
        if offload:   # the sum moves to the host between batches: the word must not keep its place on the device
            self.status = self.status.clone()
        self.offload = offload
        self._final = None
        self.stage_tokens = int(stage_tokens)
        self._stage = None   # [stage_tokens, K] bf16, allocated on first use
        self._fill = 0

    def _stream(self):
        return stream_of(self.device.index) if self.device.type == "cuda" else None

    def same_input(self, inp: torch.Tensor) -> bool:
        if self._last is None:
            return False
        t, ver = self._last
        return (t.data_ptr() == inp.data_ptr() and t.shape == inp.shape and t.stride() == inp.stride()
                and t.dtype == inp.dtype and ver == inp._version)

    def _syrk(self, x: torch.Tensor) -> None:
        if self.offload and self.H.device != self.device:
            self.H = self.H.to(self.device)
        gptq.ops.hessian_syrk(x, self.H, alpha=2.0, status=self.status)
        if self.offload:
            self.H = self.H.to("cpu")

    def flush(self) -> None:
        if self._fill:
            self._syrk(self._stage[: self._fill])
            self._fill = 0

    def accumulate(self, inp: torch.Tensor) -> None:
        if self.same_input(inp):
            return  # another member already added this batch
        x, added = gptq._tokens_2d(inp, self.device)
        t = x.shape[0]
        # (a sum that lives on the host between calls is worth fewer calls)
        if t >= (self.stage_tokens if self.offload else min(self.stage_tokens, _DIRECT_TOKENS)):
            self._syrk(x)
        else:
            if self._stage is None:
                self._stage = torch.empty((self.stage_tokens, x.shape[1]), dtype=torch.bfloat16, device=self.device)
                self._stage_home = self._stream()
            if self._fill + t > self.stage_tokens:
                self.flush()
            self._stage[self._fill: self._fill + t].copy_(x)
            self._fill += t
        self.n += added
        self._last = (inp, inp._version)

    def take_sum(self, status=None) -> torch.Tensor:
        """The lower triangle of the sum over all batches, handed over.  The status word leaves the sum's allocation, for
        ``status`` if the caller has copied it already: who reads it must not keep the matrix from being freed.
        A solve takes the sum on a stream of its own: what calibration allocated on another is not to be given out there
        before this stream has read it."""
        self._last = None
        self.flush()
        here = self._stream()
        if here != self._home or here != self._stage_home:
            stream = torch.cuda.current_stream(self.device)
            for t in (self.H, self.status, self._stage):
                if t is not None and t.is_cuda:
                    t.record_stream(stream)
        self._stage = None
        self.status = self.status.clone() if status is None else status
        H, self.H = self.H.to(self.device), None
        return H

    def finalized(self, keep: bool = False) -> torch.Tensor:
        """Full symmetric H / n.  The caller's factorisation consumes the matrix it gets;
        ``keep`` asks for a copy because another act-order setting still needs H."""
        self._last = None
        if self._final is None:
            self._final = gptq.finalize_hessian(self.take_sum(), self.n)
        out = self._final.clone() if keep else self._final
        if not keep:
            self._final = None
        return out


def _finalize_groups(groups) -> None:
    """``finalized`` for many groups: one launch for all the Hessians of a width."""
    by_width: dict = {}
    for g in groups:
        if g._final is None:
            by_width.setdefault(g.H.shape[0], []).append(g)
    for gs in by_width.values():
        if len(gs) > 1:
            for g in gs:
                g.flush()
            words = torch.cat([g.status for g in gs]).split(1)
            Hs = [g.take_sum(status) for g, status in zip(gs, words)]
            gptq.ops.hessian_finalize_many(Hs, [1.0 / g.n if g.n else 1.0 for g in gs])
            for g, H in zip(gs, Hs):
                g._final = H
