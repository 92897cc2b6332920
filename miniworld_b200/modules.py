"""Host-side mirror of the reference module interface for the triangle multiplicative update.

``TriangleMultiplication`` keeps the constructor, ``forward(pair, mask)`` signature, parameter names and
``state_dict`` layout of ``miniworld_engine.modules.TriangleMultiplication`` as MiniWorld uses it
(``src/miniworld/blocks/msa_module.py:60-71,116-117``, ``src/miniworld/blocks/template.py:41-52,84-85``
in the reference project): parameters ``ln_pair.{weight,bias}``, ``to_left``, ``to_left_gate``,
``to_right``, ``to_right_gate``, ``ln_out.{weight,bias}``, ``to_gate``, ``to_out`` (all linears
bias-free, ``benchmarks/protenix_finetune/patch_engine.py:25-29,51``); the module returns
``pair + update`` (it owns the residual).  ``TriangleMultiplicationOutgoing`` / ``...Incoming`` are the
OpenFold-style names with ``forward(z, pair_mask)``.

``BidirectionalTriangleMultiplication`` is the single operator MiniWorld's own trunk builds
(``src/miniworld/modules/mini_pairformer.py:76-80``, ``src/miniworld/modules/mini_msa_module.py:104``): one input
LayerNorm, left / right of width 2h whose halves are contracted outgoing and incoming, one LayerNorm over the 2h
contracted channels, one gate, one residual (``docs/paper/supplement.tex:125-136``); same parameter names, wider
shapes.

In training mode with ``p_drop > 0`` the forward applies the row-shared dropout of the reference
(``x + drop_row(f(x))``: one keep-mask per (batch, column, channel), shared by all rows,
``src/miniworld/blocks/template.py:38-40``). Every module here is differentiable (:mod:`miniworld_b200.training`): the triangle updates (input and all ten
parameters) and the pair Transition (input and its five parameters).
"""

from __future__ import annotations

from typing import Optional

import torch
from torch import nn

from . import _lib
from . import functional as F_

D_SUPPORTED = 128

# reference name -> OpenFold / Protenix name (benchmarks/protenix_finetune/patch_engine.py:25-29)
OPENFOLD_ALIASES = {
    "ln_pair": "layer_norm_in",
    "to_left": "linear_a_p",
    "to_left_gate": "linear_a_g",
    "to_right": "linear_b_p",
    "to_right_gate": "linear_b_g",
    "ln_out": "layer_norm_out",
    "to_gate": "linear_g",
    "to_out": "linear_z",
}

_ACCEPTED_IMPLEMENTATIONS = {None, "b200", "miniworld", "miniworld_engine", "engine", "cuda"}


def to_openfold_state_dict(sd: dict) -> dict:
    """Rename reference keys (``to_left.weight`` ...) to OpenFold keys (``linear_a_p.weight`` ...)."""
    out = {}
    for k, v in sd.items():
        head, _, tail = k.partition(".")
        out[f"{OPENFOLD_ALIASES.get(head, head)}.{tail}"] = v
    return out


def from_openfold_state_dict(sd: dict) -> dict:
    """Inverse of :func:`to_openfold_state_dict`; OpenFold bias entries of the linears are rejected."""
    inv = {v: k for k, v in OPENFOLD_ALIASES.items()}
    out = {}
    for k, v in sd.items():
        head, _, tail = k.partition(".")
        name = inv.get(head, head)
        if tail == "bias" and not name.startswith("ln_"):
            raise KeyError(f"{k}: the reference layout has bias-free linears; pass biases explicitly via set_biases()")
        out[f"{name}.{tail}"] = v
    return out


def _registered(module: nn.Module, names) -> Optional[list]:
    """The registered parameters ``"child.name"`` of ``names``, or None if one of them is not there under that name (a child
    was wrapped or re-parametrised; attribute access then says what it is). Attribute access costs about 1 us per tensor."""
    children = module._modules
    try:
        out = [children[child]._parameters[name] for child, name in names]
    except (KeyError, AttributeError):
        return None
    for t in out:
        if t is None:
            return None
    return out


class _Scratch(nn.Module):
    """A module whose scratch memory and pointer caches (``_scratch_names``) are its own: copies and pickles start without them,
    whatever a pickle of an earlier version holds."""

    _scratch_names = ()

    def __getstate__(self):
        return {**self.__dict__, **dict.fromkeys(self._scratch_names)}

    def __setstate__(self, state):
        super().__setstate__({**state, **dict.fromkeys(self._scratch_names)})


class _Kept:
    """Scratch memory that a module keeps from one call to the next, as ``(stream, tensor)`` in its attribute ``name``.

    A call takes it out of the module while it launches, so that a call from another thread does not find it, and only if the
    last call was on the same stream: on another one, that call may still be running. Otherwise the call allocates its own, which
    replaces the kept one (its memory goes back to the allocator, in the order of the stream it was allocated on). A call that is
    being captured never takes kept memory, and what it allocates, in the graph's pool, is not taken again (stream -1)."""

    def __init__(self, module: nn.Module, name: str, need: int, device: torch.device, clear=None):
        self.module, self.name, self.need, self.device, self.clear = module, name, need, device, clear

    def __enter__(self) -> torch.Tensor:
        kept = self.module.__dict__.pop(self.name, None)
        with torch.cuda.device(self.device):
            stream = -1 if torch.cuda.is_current_stream_capturing() else torch.cuda.current_stream().cuda_stream
        if kept is None or stream < 0 or kept[0] != stream or kept[1].device != self.device or kept[1].numel() < self.need:
            kept = (stream, F_.aligned_empty(self.need, self.device))
            if self.clear is not None:
                self.clear(kept[1])
        self.kept = kept
        return kept[1]

    def __exit__(self, *error) -> None:
        self.module.__dict__[self.name] = self.kept


class Fp32LayerNorm(nn.LayerNorm):
    """LayerNorm parameter holder whose affine parameters are pinned to fp32: ``module.to(torch.bfloat16)`` moves them
    between devices but never changes (or rounds) their values, like the reference's fp32-pinned LayerNorm
    (``src/miniworld/layers/primitives.py:86-88``). Only ``weight``, ``bias`` and ``eps`` are used; the
    normalisation itself runs inside the fused kernels."""

    def _apply(self, fn, recurse=True):
        def pinned(t):
            out = fn(t)
            if t.is_floating_point() and out.dtype != t.dtype:
                return t.to(device=out.device)  # follow the device, keep the fp32 values bit for bit
            return out

        return super()._apply(pinned, recurse)


_TRI_NAMES = tuple(tuple(k.split(".")) for k in (
    "ln_pair.weight", "ln_pair.bias", "to_left.weight", "to_left_gate.weight", "to_right.weight", "to_right_gate.weight",
    "ln_out.weight", "ln_out.bias", "to_gate.weight", "to_out.weight"))
_TRANSITION_NAMES = tuple(tuple(k.split(".")) for k in F_.TRANSITION_KEYS)


class TriangleMultiplication(_Scratch):
    """Triangle multiplicative update on B200 kernels (forward and backward).

    ``forward(pair [B,N,N,d_pair] bf16, mask Bool[B,N] | None) -> pair + update`` (bf16).
    Linear weights may be bf16 or fp32 masters; LayerNorm affine parameters are kept in fp32 whatever
    ``.to(dtype)`` is applied to the module (``src/miniworld/layers/primitives.py:86-88``).
    ``ln_pair.eps`` / ``ln_out.eps`` are read at call time.
    """

    _bidirectional = False
    _scratch_names = ("_workspace", "_wcache")

    def __init__(
        self,
        d_pair: int,
        d_hidden: Optional[int] = None,
        outgoing: bool = True,
        implementation=None,
        p_drop: float = 0.0,
        residual: bool = True,
        check_status: bool = False,
    ):
        super().__init__()
        wide = 2 if self._bidirectional else 1
        d_hidden = d_pair if d_hidden is None else d_hidden
        # the kernels contract 128 channels per call of the contraction stage and take 128 or 64 input channels:
        #   d_pair 128, d_hidden 128 (either module);  d_pair 64 with d_hidden 128 (one direction: the template
        #   blocks of the Protenix harness, benchmarks/protenix_finetune/patch_engine.py:283-295);  d_pair 64 with
        #   d_hidden 64 (bidirectional: the (L, D) = (384, 64) case of the reference's validation,
        #   docs/archive/engine2-validation-20260923/validate_bidir_reference.py:11)
        ok = (d_pair, d_hidden) == (D_SUPPORTED, D_SUPPORTED) or (d_pair, wide * d_hidden) == (64, D_SUPPORTED)
        if not ok:
            raise NotImplementedError(
                f"implemented widths: d_pair = d_hidden = {D_SUPPORTED}; d_pair = 64 with d_hidden = 128 (one direction) or "
                f"64 (bidirectional); got d_pair = {d_pair}, d_hidden = {d_hidden}"
            )
        if d_pair != D_SUPPORTED and p_drop > 0.0:
            raise NotImplementedError("the row-shared dropout of the training forward is only implemented for d_pair = 128")
        impl = getattr(implementation, "value", implementation)
        impl = impl.lower() if isinstance(impl, str) else impl
        if impl not in _ACCEPTED_IMPLEMENTATIONS:
            raise ValueError(f"implementation={implementation!r}: this module has exactly one backend (B200 CUDA kernels)")
        self.d_pair = d_pair
        self.d_hidden = d_hidden
        self.outgoing = bool(outgoing)
        self.p_drop = float(p_drop)
        self.residual = bool(residual)
        self.check_status = bool(check_status)
        self.ln_pair = Fp32LayerNorm(d_pair, eps=1e-5)
        self.to_left = nn.Linear(d_pair, wide * d_hidden, bias=False)
        self.to_left_gate = nn.Linear(d_pair, wide * d_hidden, bias=False)
        self.to_right = nn.Linear(d_pair, wide * d_hidden, bias=False)
        self.to_right_gate = nn.Linear(d_pair, wide * d_hidden, bias=False)
        self.ln_out = Fp32LayerNorm(wide * d_hidden, eps=1e-5)
        self.to_gate = nn.Linear(d_pair, d_pair, bias=False)
        self.to_out = nn.Linear(wide * d_hidden, d_pair, bias=False)
        # the reference initialises the two output linears to zero ("init='zero'")
        nn.init.zeros_(self.to_gate.weight)
        nn.init.zeros_(self.to_out.weight)
        self._biases: Optional[dict] = None
        self._workspace: Optional[tuple] = None  # (stream, workspace) of the last forward, see _Kept
        self._wcache = None  # (key, validated parameter pointers); the values themselves are re-read every call

    # ------------------------------------------------------------------ dtype handling
    def _apply(self, fn, recurse=True):
        super()._apply(fn, recurse)  # the LayerNorm affine parameters stay fp32 (Fp32LayerNorm)
        self._workspace = None
        self._wcache = None
        return self

    def set_biases(self, biases: Optional[dict]) -> None:
        """Optional fp32[d] biases for the linears, keys ``to_left`` ... ``to_out`` (None = reference layout).

        They are not parameters and are not part of the ``state_dict`` (the reference module has none).
        """
        self._biases = None if not biases else dict(biases)
        self._wcache = None

    def _weights(self, device: torch.device):
        """Validated parameter pointers, rebuilt only when a parameter tensor was replaced, moved or re-typed."""
        params = self._params()
        key = tuple((v.data_ptr(), v.dtype, v.device, v.is_contiguous()) for v in params.values()) + (device,)
        if self._wcache is None or self._wcache[0] != key:
            self._wcache = (key, F_._Weights(params, self._biases, device, bidirectional=self._bidirectional,
                                             d_pair=self.d_pair))
        return self._wcache[1]

    def _params(self) -> dict:
        return {
            "ln_pair.weight": self.ln_pair.weight,
            "ln_pair.bias": self.ln_pair.bias,
            "to_left.weight": self.to_left.weight,
            "to_left_gate.weight": self.to_left_gate.weight,
            "to_right.weight": self.to_right.weight,
            "to_right_gate.weight": self.to_right_gate.weight,
            "ln_out.weight": self.ln_out.weight,
            "ln_out.bias": self.ln_out.bias,
            "to_gate.weight": self.to_gate.weight,
            "to_out.weight": self.to_out.weight,
        }

    def load_openfold_state_dict(self, sd: dict, strict: bool = True):
        return self.load_state_dict(from_openfold_state_dict(sd), strict=strict)

    def device_status(self) -> int:
        """Synchronise and return the device status word of the last forward: 0, or the 1xx code of a device-side wait
        that gave up (:func:`miniworld_b200.functional.check_status` raises on it)."""
        kept = self.__dict__.get("_workspace")
        return 0 if kept is None else F_.read_status(kept[1][:64].view(torch.int32))

    def _direction(self):
        return None if self._bidirectional else self.outgoing

    def _make_drop_row_scale(self, pair: torch.Tensor, p: float) -> torch.Tensor:
        """Row-shared dropout scale [B, 1, N, C]: keep-mask / (1 - p), one draw per (batch, column, channel), shared by
        all rows (the reference's hook of the same name, ``scripts/check_trimul_module_reference.py:43,100-103``;
        tests replace it to fix the mask)."""
        B, N, C = pair.shape[0], pair.shape[2], pair.shape[3]
        keep = torch.rand(B, 1, N, C, device=pair.device) >= p
        return keep.to(torch.bfloat16) / (1.0 - p)

    def _backward_supported(self) -> bool:
        return True  # every width the constructor accepts has a backward

    def _run(self, pair: torch.Tensor, token_mask, pair_mask) -> torch.Tensor:
        # the differentiable path is taken when the input requires grad, or in training mode when a parameter does
        train = torch.is_grad_enabled() and (
            pair.requires_grad or (self.training and any(q.requires_grad for q in self.parameters()))
        )
        if not train and self._biases is None and not self.check_status and not (self.training and self.p_drop > 0.0):
            y = self._run_native(pair, token_mask, pair_mask)
            if y is not None:
                return y
        if train and not self._backward_supported():
            if pair.requires_grad:
                raise NotImplementedError(
                    "backward is implemented for d_pair = d_hidden = 128 only: call under "
                    "torch.no_grad() or with an input that does not require grad"
                )
            train = False
        if pair.dim() != 4 or pair.shape[1] != pair.shape[2] or pair.shape[3] != self.d_pair:
            raise RuntimeError(f"pair must be [B, N, N, {self.d_pair}], got {tuple(pair.shape)}")
        if not pair.is_cuda:
            raise RuntimeError("pair must be a CUDA tensor: this module has no CPU implementation")
        in_dtype = pair.dtype
        if train:
            return self._run_train(pair, token_mask, pair_mask)
        z = pair.detach()
        if z.dtype != torch.bfloat16:
            z = z.to(torch.bfloat16)
        z = z.contiguous()
        B, N = int(z.shape[0]), int(z.shape[1])
        ragged = N % 8 != 0
        scale = None
        if self.training and self.p_drop > 0.0:
            scale = self._make_drop_row_scale(z, self.p_drop).to(device=z.device, dtype=torch.bfloat16)
        if ragged:
            # any length runs as it is; masks and scale may be given in a form that broadcasts to the batch
            z = F_.aligned16(z)
            if token_mask is not None:
                token_mask = torch.broadcast_to(token_mask.to(z.device), (B, N))
            if pair_mask is not None:
                pair_mask = torch.broadcast_to(pair_mask.to(z.device), (B, N, N))
            if scale is not None:
                scale = F_.aligned16(torch.broadcast_to(scale, (B, 1, N, self.d_pair)).contiguous())
        need = F_._forward_need(B, F_._pitch(N) if ragged else N, self._direction(), self.d_pair)
        with torch.no_grad(), _Kept(self, "_workspace", need, z.device) as workspace:
            y = F_._forward(
                z, self._params(), token_mask, self._direction(), float(self.ln_pair.eps), float(self.ln_out.eps), pair_mask,
                self.residual, self._biases, workspace, None, self.check_status, self._weights(z.device), scale, ragged,
            )
        return y if in_dtype == torch.bfloat16 else y.to(in_dtype)

    def _run_native(self, pair, token_mask, pair_mask) -> Optional[torch.Tensor]:
        """The forward without a graph as one native call, or None for a call that needs converting or refusing."""
        from .training import ordinary

        if not ordinary(pair) or pair.dim() != 4:
            return None
        children = self._modules  # (attribute access costs 0.3 us per child, and 1 us more per parameter)
        eps_in, eps_out = (getattr(children.get(k), "eps", None) for k in ("ln_pair", "ln_out"))
        if eps_in is None or eps_out is None:
            return None
        kept = self.__dict__.pop("_workspace", None)  # (see _Kept)
        got = _lib.native().trimul_forward(
            pair, (children, _TRI_NAMES), token_mask, pair_mask, kept, self.d_pair, F_._direction(self._direction()), eps_in,
            eps_out, self.residual, pair.shape[1] % 8 != 0,
        )
        if got is None:
            self.__dict__["_workspace"] = kept
            return None
        y, self.__dict__["_workspace"] = got
        return y

    def _run_train(self, pair: torch.Tensor, token_mask, pair_mask) -> torch.Tensor:
        """Differentiable forward (:mod:`miniworld_b200.training`): the stage tensors of this call are kept for the
        backward in a workspace of their own; dtype casts are ordinary differentiable ops."""
        from .training import _PARAM_KEYS, _trimul_train

        in_dtype = pair.dtype
        z = pair if pair.dtype == torch.bfloat16 else pair.to(torch.bfloat16)
        z = z.contiguous()
        B, N = int(z.shape[0]), int(z.shape[1])
        ragged = N % 8 != 0
        scale = None
        if self.training and self.p_drop > 0.0:
            scale = self._make_drop_row_scale(z, self.p_drop).to(device=z.device, dtype=torch.bfloat16).contiguous()
        if ragged:
            # any length runs as it is. What the backward reads is this call's own (a caller may change the pair tensor or
            # the masks in place between the two passes of such a length)
            if z is pair:
                z = z.clone()
            if token_mask is not None:
                token_mask = token_mask.to(z.device) != 0
            if pair_mask is not None:
                pair_mask = pair_mask.to(z.device) != 0
            if scale is not None:
                scale = F_.aligned16(scale)
        plain = _registered(self, _TRI_NAMES)
        params = self._params() if plain is None else dict(zip(_PARAM_KEYS, plain))
        y = _trimul_train(z, params, token_mask, self._direction(), float(self.ln_pair.eps), float(self.ln_out.eps),
                          pair_mask, self.residual, self._biases, scale, self.check_status, ragged)
        return y if in_dtype == torch.bfloat16 else y.to(in_dtype)

    def forward(self, pair: torch.Tensor, mask: Optional[torch.Tensor] = None) -> torch.Tensor:
        if mask is not None and mask.dim() != 2:
            raise RuntimeError(f"mask must be a token mask [B, N], got {tuple(mask.shape)}")
        return self._run(pair, mask, None)


class _OpenFoldStyle(TriangleMultiplication):
    """``forward(z, pair_mask)`` where ``pair_mask`` is None, a token mask [B,N] or a pair mask [B,N,N]."""

    _outgoing = True

    def __init__(self, d_pair: int = D_SUPPORTED, d_hidden: Optional[int] = None, residual: bool = True, **kw):
        kw.pop("outgoing", None)
        super().__init__(d_pair, d_hidden, outgoing=self._outgoing, residual=residual, **kw)

    def forward(self, z: torch.Tensor, pair_mask: Optional[torch.Tensor] = None) -> torch.Tensor:
        if pair_mask is None or pair_mask.dim() == 2:
            return self._run(z, pair_mask, None)
        if pair_mask.dim() == 3:
            return self._run(z, None, pair_mask)
        raise RuntimeError(f"pair_mask must be [B,N] or [B,N,N], got {tuple(pair_mask.shape)}")


class TriangleMultiplicationOutgoing(_OpenFoldStyle):
    _outgoing = True


class TriangleMultiplicationIncoming(_OpenFoldStyle):
    _outgoing = False


class BidirectionalTriangleMultiplication(TriangleMultiplication):
    """Both directions in one operator: ``forward(pair [B,N,N,128] bf16, mask Bool[B,N] | None) -> pair + update``.

    Constructor as in the reference (``BidirectionalTriangleMultiplication(d_pair, implementation=..., p_drop=...)``,
    ``src/miniworld/modules/mini_pairformer.py:76-80``). Parameters: ``ln_pair`` [128]; ``to_left``, ``to_left_gate``,
    ``to_right``, ``to_right_gate`` [256, 128] (rows 0-127: outgoing half, rows 128-255: incoming half); ``ln_out``
    [256]; ``to_gate`` [128, 128]; ``to_out`` [128, 256].
    """

    _bidirectional = True

    def __init__(self, d_pair: int = D_SUPPORTED, d_hidden: Optional[int] = None, implementation=None, p_drop: float = 0.0,
                 residual: bool = True, check_status: bool = False):
        super().__init__(d_pair, d_hidden, outgoing=True, implementation=implementation, p_drop=p_drop,
                         residual=residual, check_status=check_status)


class Transition(_Scratch):
    """Pair transition ``x + squeeze(SiLU(expand_a(LN x)) * expand_b(LN x))`` on the B200 kernels (forward and backward).

    Mirrors ``miniworld_engine.modules.Transition(d, n=4, implementation=...)`` as MiniWorld's blocks build it
    (``src/miniworld/modules/mini_pairformer.py:81-84``; it owns its residual, ``:108``): parameters ``ln_in`` [d],
    ``expand_a`` / ``expand_b`` [n d, d], ``squeeze`` [d, n d], all linears bias-free
    (``benchmarks/protenix_finetune/patch_engine.py:35-37``). d = 128 and n = 4 are what the kernel takes.
    """

    _scratch_names = ("_scratch",)

    def __init__(self, d: int = D_SUPPORTED, n: int = 4, implementation=None, residual: bool = True, check_status: bool = False):
        super().__init__()
        if d != D_SUPPORTED or n != 4:
            raise NotImplementedError(f"only d = {D_SUPPORTED}, n = 4 is implemented on this path (got d = {d}, n = {n})")
        impl = getattr(implementation, "value", implementation)
        impl = impl.lower() if isinstance(impl, str) else impl
        if impl not in _ACCEPTED_IMPLEMENTATIONS:
            raise ValueError(f"implementation={implementation!r}: this module has exactly one backend (B200 CUDA kernels)")
        self.d, self.n = d, n
        self.residual = bool(residual)
        self.check_status = bool(check_status)
        self.ln_in = Fp32LayerNorm(d, eps=1e-5)
        self.expand_a = nn.Linear(d, n * d, bias=False)
        self.expand_b = nn.Linear(d, n * d, bias=False)
        self.squeeze = nn.Linear(n * d, d, bias=False)
        nn.init.zeros_(self.squeeze.weight)  # the reference's final linears start at zero
        self._scratch = None  # (stream, packed weights and status words) of the last forward without a graph, see _Kept

    def _apply(self, fn, recurse=True):
        super()._apply(fn, recurse)
        self._scratch = None
        return self

    def device_status(self) -> int:
        kept = self.__dict__.get("_scratch")
        return 0 if kept is None else F_.read_status(self._split(kept[1])[1])

    def _run_native(self, x: torch.Tensor) -> Optional[torch.Tensor]:
        """The forward without a graph as one native call, or None for a call that needs converting or refusing."""
        eps = getattr(self._modules.get("ln_in"), "eps", None)
        if eps is None:
            return None
        kept = self.__dict__.pop("_scratch", None)  # (see _Kept)
        got = _lib.native().transition_forward(x, (self._modules, _TRANSITION_NAMES), kept, eps, self.residual)
        if got is None:
            self.__dict__["_scratch"] = kept
            return None
        y, self.__dict__["_scratch"] = got
        return y

    @staticmethod
    def _split(scratch: torch.Tensor):
        n = F_.transition_packed_bytes()
        return scratch[:n], scratch[n : n + 64].view(torch.int32)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        from .training import ordinary, transition_train

        if not x.is_cuda:
            raise RuntimeError("input must be a CUDA tensor: this module has no CPU implementation")
        if x.shape[-1] != self.d:
            raise RuntimeError(f"input must be [..., {self.d}], got {tuple(x.shape)}")
        in_dtype = x.dtype
        # the differentiable path is taken when the input requires grad, or in training mode when a parameter does
        train = torch.is_grad_enabled() and (x.requires_grad or (self.training and any(q.requires_grad for q in self.parameters())))
        if not train and not self.check_status and in_dtype == torch.bfloat16 and ordinary(x):
            y = self._run_native(x)
            if y is not None:
                return y
        plain = _registered(self, _TRANSITION_NAMES)
        params = dict(zip(F_.TRANSITION_KEYS, plain)) if plain is not None else {
            "ln_in.weight": self.ln_in.weight, "ln_in.bias": self.ln_in.bias, "expand_a.weight": self.expand_a.weight,
            "expand_b.weight": self.expand_b.weight, "squeeze.weight": self.squeeze.weight}
        if train:
            xb = (x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)).contiguous()
            y = transition_train(xb, params, eps=float(self.ln_in.eps), residual=self.residual, check=self.check_status)
            return y if in_dtype == torch.bfloat16 else y.to(in_dtype)
        xb = x.detach()
        if xb.dtype != torch.bfloat16:
            xb = xb.to(torch.bfloat16)
        xb = xb.contiguous()
        if not x.is_contiguous() and not self.check_status and in_dtype == torch.bfloat16 and ordinary(x):
            y = self._run_native(xb)
            if y is not None:
                return y
        clear = lambda t: self._split(t)[1].zero_()  # noqa: E731
        with torch.no_grad(), _Kept(self, "_scratch", F_.transition_packed_bytes() + 64, xb.device, clear) as scratch:
            packed, status = self._split(scratch)
            F_.transition_pack_weights(params, packed)  # packed in every call: a captured graph replays current weights
            y = F_.transition_forward(xb, packed, status, eps=float(self.ln_in.eps), residual=self.residual)
            if self.check_status:
                F_.check_status(status, "b200_transition_forward")
        return y if in_dtype == torch.bfloat16 else y.to(in_dtype)
