"""Multi-head module around the sliding-window 2-simplicial attention operator.

``SlidingWindowTwoSimplicialMHA`` keeps the constructor, forward signature and
``state_dict`` keys of the reference module
(simplicial_attention/triton_two_simplicial_attention.py:1062-1081, built on
``HigherOrderAttention``, simplicial_attention/simplicial_mha.py:28-138), so
checkpoints of the reference load unchanged:
``q_norm.weight, k_norms.{0,1}.weight, v_norms.{0,1}.weight, to_qkv.weight,
combine_heads.weight`` (+ ``prenorm.weight`` / ``postnorm.weight`` when on).

The projections and norms are plain PyTorch; only ``attend`` is ours.
"""
from __future__ import annotations

from functools import partial
from typing import Callable

import torch
from torch.nn import Identity, Linear, Module, ModuleList, RMSNorm
from torch.nn.modules.module import _has_any_global_hook

from . import _lib
from .attention import divisible_by, exists, sliding_two_simplicial_attn
from .headnorm import RMSNorm as RowRMSNorm


def default(v, d):
    return v if exists(v) else d


def _child(module, name):
    """``module.name`` for a submodule or parameter, from the module's own tables where it is there: torch's attribute lookup
    costs a generation step of one sequence, which the host bounds, a third of a microsecond each."""
    d = module.__dict__
    found = d["_modules"].get(name)
    if found is None:
        found = d["_parameters"].get(name)
    return getattr(module, name) if found is None else found


class HigherOrderAttention(Module):
    """Projection / head-split / norm shell with a pluggable ``attend``
    callable ``attend(queries, keys, values[, causal=True]) -> out``
    (simplicial_mha.py:41,97-103,131)."""

    def __init__(
        self,
        dim,
        causal=False,
        dim_head=64,
        dim_head_values=None,
        heads=8,
        key_value_heads=None,
        number_key_value_sets=2,
        qk_rmsnorm=True,
        prenorm=False,
        postnorm=False,
        attend: Callable | None = None,
        head_first_dim=True,
    ):
        super().__init__()
        if not exists(attend):
            raise ValueError("pass attend=..., or use SlidingWindowTwoSimplicialMHA: this package ships only "
                             "the sliding-window 2-simplicial attend")
        self.causal = causal
        self.scale = dim_head ** -0.5
        self.heads = heads
        self.key_value_heads = default(key_value_heads, heads)
        assert divisible_by(heads, self.key_value_heads)
        self.query_head_groups = heads // self.key_value_heads
        self.dim_head = dim_head
        self.dim_head_values = default(dim_head_values, dim_head)
        self.kv_sets = number_key_value_sets
        self.head_first_dim = head_first_dim

        # same parameter as torch.nn.RMSNorm; one fused kernel on CUDA
        self.prenorm = RowRMSNorm(dim) if prenorm else Identity()
        self.postnorm = RowRMSNorm(dim) if postnorm else Identity()

        self.qk_rmsnorm = qk_rmsnorm
        if qk_rmsnorm:
            self.q_norm = RMSNorm(dim_head)
            self.k_norms = ModuleList([RMSNorm(dim_head) for _ in range(self.kv_sets)])
            self.v_norms = ModuleList([RMSNorm(dim_head) for _ in range(self.kv_sets)])

        self.split_dims = (
            heads * dim_head,
            self.kv_sets * self.key_value_heads * dim_head,
            self.kv_sets * self.key_value_heads * self.dim_head_values,
        )
        self.to_qkv = Linear(dim, sum(self.split_dims), bias=False)

        if causal:
            attend = partial(attend, causal=causal)
        self.attend = attend

        self.combine_heads = Linear(heads * self.dim_head_values, dim, bias=False)

    def _split(self, t, heads):
        b, n, _ = t.shape
        t = t.view(b, n, heads, -1)
        return t.transpose(1, 2) if self.head_first_dim else t

    # One kernel normalises the whole fused projection instead of five RMSNorm modules plus casts
    # (CUDA tensors only; set to False to run the norms as separate torch modules, as the reference does).
    fused_head_norm = True
    # Wider projections use the separate modules where there may be a backward, whose kernel spans a row with one CTA (25
    # warps of 256 channels).  May be lowered, never raised.  Generation has no such limit.
    fused_head_norm_max_channels = 6400

    def _fused_norm(self, proj):
        """Per-head RMSNorm of the packed projection with the gains of q_norm / k_norms / v_norms tiled to
        one entry per channel; same arithmetic as the modules, applied before the split."""
        from .headnorm import head_rmsnorm
        kw = torch.cat([n.weight for n in self.k_norms]).repeat(self.key_value_heads)
        vw = torch.cat([n.weight for n in self.v_norms]).repeat(self.key_value_heads)
        weight = torch.cat((self.q_norm.weight.repeat(self.heads), kw, vw))
        autocast = torch.is_autocast_enabled()
        # the modules leave eps unset: the machine epsilon of the dtype they compute in (fp32 under autocast)
        eps = self.q_norm.eps if self.q_norm.eps is not None else \
            torch.finfo(torch.float32 if autocast else proj.dtype).eps
        out_dtype = torch.get_autocast_dtype("cuda") if autocast else proj.dtype
        return head_rmsnorm(proj, weight, self.dim_head, eps, out_dtype)

    def _project(self, tokens):
        """tokens -> (queries, keys, values) after the head split and the per-head norms."""
        return self._split_heads(self.to_qkv(self.prenorm(tokens)))

    def _split_heads(self, proj):
        fused = (self.fused_head_norm and self.qk_rmsnorm and proj.is_cuda and not self.head_first_dim
                 and self.dim_head_values == self.dim_head and self.dim_head in (32, 64, 128)
                 and proj.shape[-1] <= self.fused_head_norm_max_channels
                 and proj.dtype in (torch.float32, torch.bfloat16))
        if fused:
            q, k, v = self._fused_norm(proj).split(self.split_dims, dim=-1)
            queries = self._split(q, self.heads)
            keys = self._split(k, self.key_value_heads).chunk(self.kv_sets, dim=-1)
            values = self._split(v, self.key_value_heads).chunk(self.kv_sets, dim=-1)
            return queries, keys, values
        q, k, v = proj.split(self.split_dims, dim=-1)

        queries = self._split(q, self.heads)
        # each kv head's slice holds its key sets side by side: [k1 | k2]
        keys = self._split(k, self.key_value_heads).chunk(self.kv_sets, dim=-1)
        values = self._split(v, self.key_value_heads).chunk(self.kv_sets, dim=-1)

        if self.qk_rmsnorm:
            queries = self.q_norm(queries)
            keys = tuple(norm(t) for norm, t in zip(self.k_norms, keys))
            values = tuple(norm(t) for norm, t in zip(self.v_norms, values))
        return queries, keys, values

    def _merge(self, out):
        if self.head_first_dim:
            out = out.transpose(1, 2)
        out = out.reshape(out.shape[0], out.shape[1], -1)
        return self.postnorm(self.combine_heads(out))

    def forward(self, tokens):
        queries, keys, values = self._project(tokens)
        return self._merge(self.attend(queries, keys, values))


class SlidingWindowTwoSimplicialMHA(HigherOrderAttention):
    def __init__(self, *args, w1=512, w2=32, **kwargs):
        assert "number_key_value_sets" not in kwargs
        assert "head_first_dim" not in kwargs
        # the kernels contract q, k, k' and aggregate v, v' over one head dimension; say so at construction
        # instead of failing at the first forward (the reference accepts the argument, simplicial_mha.py:34,
        # and then fails inside its kernels, which read values with the key head dim)
        dim_head = kwargs.get("dim_head", args[2] if len(args) > 2 else 64)
        dim_head_values = kwargs.get("dim_head_values", args[3] if len(args) > 3 else None)
        if dim_head_values is not None and dim_head_values != dim_head:
            raise ValueError(f"dim_head_values ({dim_head_values}) must equal dim_head ({dim_head}) for the "
                             "sliding-window 2-simplicial kernels")
        attend = partial(sliding_two_simplicial_attn, w1=w1, w2=w2, causal=True)
        super().__init__(*args, number_key_value_sets=2, head_first_dim=False, attend=attend, **kwargs)
        self.w1, self.w2 = w1, w2

    def _fused_call(self, proj):
        """Arguments of the native calls that take the packed projection as a whole - norm and attention, forward and
        backward, without splitting or concatenating it - or None where the general path is needed.  ``proj`` is the
        projection, or tokens of its device and dtype."""
        at = self.attend
        if not (self.fused_head_norm and self.qk_rmsnorm and proj.is_cuda and isinstance(at, partial)
                and at.func is sliding_two_simplicial_attn and not at.args
                and at.keywords.keys() <= {"w1", "w2", "causal", "kernel"} and at.keywords.get("causal", True)):
            return None
        autocast = torch.is_autocast_enabled()
        norms = [_child(self, "q_norm"), *_child(self, "k_norms")._modules.values(), *_child(self, "v_norms")._modules.values()]
        eps = norms[0].eps
        for n in norms:
            if n.eps != eps:
                return None
        # the modules leave eps unset: the machine epsilon of the dtype they compute in (fp32 under autocast)
        if eps is None:
            eps = torch.finfo(torch.float32 if autocast else proj.dtype).eps
        dtype = torch.get_autocast_dtype("cuda") if autocast else proj.dtype
        return ([_child(n, "weight") for n in norms], (self.heads, self.key_value_heads, self.dim_head, eps), dtype,
                (at.keywords.get("w1", 512), at.keywords.get("w2", 32), _lib.KERNELS[at.keywords.get("kernel", "auto")]))

    def _attend_packed(self, tokens):
        """The attention output before the heads are combined, or the projection when the general path has to run."""
        proj = self.to_qkv(self.prenorm(tokens))
        call = self._fused_call(proj)
        if call is None:
            return proj, None
        if proj.shape[-1] > self.fused_head_norm_max_channels:
            return proj, None
        gains, heads, dtype, windows = call
        return proj, _lib.ext().qkv_attn(proj, gains, *heads, dtype, *windows)

    def _step(self, tokens, cache):
        """A generation step as one native call, or None where a submodule is not the plain one this class made
        (another type, a hook, a bias) or autocast is on: then the modules are called one by one."""
        pre, post, qkv, comb = [_child(self, name) for name in ("prenorm", "postnorm", "to_qkv", "combine_heads")]
        norms = (RowRMSNorm, Identity)
        if type(pre) not in norms or type(post) not in norms or type(qkv) is not Linear or type(comb) is not Linear \
                or qkv._parameters.get("bias", qkv) is not None or comb._parameters.get("bias", comb) is not None or torch.is_autocast_enabled() or _has_any_global_hook():
            return None
        for m in (pre, post, qkv, comb):
            if m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__:
                return None
        call = self._fused_call(tokens)
        if call is None or call[3][:2] != (self.w1, self.w2):
            return None
        gains, heads, dtype, windows = call
        args = [(None, 0.) if type(m) is Identity else (_child(m, "weight"), m.eps if m.eps is not None else torch.finfo(dtype).eps) for m in (pre, post)]
        return _lib.ext().step(tokens, *args[0], _child(qkv, "weight"), gains, [*cache[0], *cache[1]], *heads, *windows, _child(comb, "weight"), *args[1])

    def forward(self, tokens, cache=None, return_cache=False):
        """``cache`` (from an earlier call with ``return_cache=True``) holds the last ``w1 - 1`` rows of the
        first key/value set and the last ``w2 - 1`` rows of the second: all a later token can still see.
        With a cache, ``tokens`` are only the new positions; the cached rows ride in front of the new keys
        as the halo the kernels already understand, so decoding a token costs one window, not the prefix
        (the reference's sampling loop re-runs the whole prefix for every token, train.py:103-104)."""
        if cache is None and not return_cache:
            proj, out = self._attend_packed(tokens)
            if out is not None:
                return self._merge(out)
            queries, keys, values = self._split_heads(proj)
            return self._merge(self.attend(queries, keys, values))
        generating = cache is not None and return_cache and not torch.is_grad_enabled()
        if generating:
            res = self._step(tokens, cache)
            if res is not None:
                return res[0], ((res[1], res[2]), (res[3], res[4]))
        proj = self.to_qkv(self.prenorm(tokens))
        if generating:
            call = self._fused_call(proj)
            if call is not None and call[2] == proj.dtype and call[3][:2] == (self.w1, self.w2):
                gains, heads, _, windows = call
                res = _lib.ext().qkv_attn_cached(proj, gains, [*cache[0], *cache[1]], *heads, *windows)
                if res is not None:
                    return self._merge(res[0]), ((res[1], res[2]), (res[3], res[4]))
        queries, keys, values = self._split_heads(proj)
        if cache is not None:
            keys = tuple(torch.cat((c, t), dim=1) for c, t in zip(cache[0], keys))
            values = tuple(torch.cat((c, t), dim=1) for c, t in zip(cache[1], values))
        out = self._merge(self.attend(queries, keys, values))
        if not return_cache:
            return out
        keep = (self.w1 - 1, self.w2 - 1)
        new_cache = (tuple(t[:, t.shape[1] - min(k, t.shape[1]):].detach() for t, k in zip(keys, keep)),
                     tuple(t[:, t.shape[1] - min(k, t.shape[1]):].detach() for t, k in zip(values, keep)))
        return out, new_cache
