"""The two layer types whose forward pass chooses among the quantized matmuls: the host-side mirror of the
reference's nn.Linear (nn/linear.go:193-354, 476-516) and nn.SparseMoE (nn/moe.go:121-245).

They carry no kernels of their own.  Each forward checks what the reference checks, in the reference's words, and
dispatches to one `ops` call per weight kind:

    weight                       call                       reference branch
    GGUF block-quantized         ops.MatMulQ                nn/linear.go:273-280
    4-bit GPTQ / AWQ (W4)        ops.MatMulInt4             nn/linear.go:476-516
    FP8 with block scales        ops.MatMulF8Block          nn/linear.go:255-258
    F32 / BF16 / F16             the library GEMM           nn/linear.go:300-330

The dense branch is a plain library GEMM on the device, as it is in the reference (cuBLAS); everything else is this
package's own kernels.  LoRA adapters, autograd and per-tensor FP8 (the cuBLASLt FP8 GEMM) are outside this path.
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Callable, Optional, Sequence, Tuple, Union

import torch

from . import ops


@dataclass
class Linear:
    """y = x @ W^T + b.  Exactly one of `W` (dense tensor or ops.QTensor) and `W4` (ops.Int4) is set."""
    in_features: int
    out_features: int
    W: Union[torch.Tensor, ops.QTensor, None] = None
    B: Optional[torch.Tensor] = None
    W4: Optional[ops.Int4] = None
    WBlockScale: Optional[torch.Tensor] = None
    WBlock: Tuple[int, int] = (0, 0)

    def set_weight(self, w) -> None:
        """Linear.SetWeight: shape-checked install of a dense or block-quantized weight."""
        shape = tuple(w.shape)
        if shape != (self.out_features, self.in_features):
            raise ValueError(f"nn.Linear.SetWeight: weight {shape}, want ({self.out_features}, {self.in_features})")
        self.W, self.W4 = w, None

    def set_int4(self, w: ops.Int4) -> None:
        """Linear.SetInt4."""
        if (w.N(), w.K()) != (self.out_features, self.in_features):
            raise ValueError(f"nn.Linear.SetInt4: weight ({w.N()}, {w.K()}), want ({self.out_features}, {self.in_features})")
        self.W4, self.W = w, None

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        w = self.W
        if self.B is None:  # the common forms as one native call; None: not one of them, or an error to be named below
            y, w4 = None, self.W4
            if w4 is not None:
                if w4.perm is None and x.dim() and x.shape[-1] == self.in_features and w4.codes.shape[0] == self.out_features:
                    y = ops._host.linear_int4(x, w4.codes, w4.scales, w4.zeros, w4.group)
            elif type(w) is ops.QTensor:
                if w.shape == (self.out_features, self.in_features):
                    y = ops._host.linear_q(x, w.data, w.ggml_type, self.out_features, self.in_features)
            elif w is not None and w.dtype is torch.float8_e4m3fn and self.WBlockScale is not None and x.dim() and x.shape[-1] == self.in_features and \
                    w.shape[0] == self.out_features:
                y = ops._host.linear_f8(x, w, self.WBlockScale, *self.WBlock)
            if y is not None:
                return y
        if self.W4 is not None:
            return self._forward_int4(x)
        if self.W is None:
            raise ValueError(f"nn.Linear: weight not loaded (placeholder layer {self.in_features}→{self.out_features})")
        wdev = self.W.device
        if x.device != wdev:
            raise ValueError(f"nn.Linear: x on {x.device} but W on {wdev}")
        if x.dim() < 1 or x.shape[-1] != self.in_features:
            raise ValueError(f"nn.Linear: last dim of x ({x.shape[-1] if x.dim() else 0}) != in_features ({self.in_features})")
        quantized = isinstance(self.W, ops.QTensor)
        if quantized and x.dtype != torch.float32:
            raise ValueError(f"nn.Linear: quantized weight ({ops.GGUF_NAMES[self.W.ggml_type]}) needs F32 activations, got {x.dtype}")
        fp8 = (not quantized) and self.W.dtype == torch.float8_e4m3fn
        if fp8 and self.WBlockScale is None:
            raise ValueError("nn.Linear: per-tensor FP8 weights run the library's FP8 GEMM in the reference; only block-scaled FP8 is built here")
        if fp8 and x.dtype == torch.float16:
            raise ValueError("nn.Linear: block-scaled FP8 needs F32 or BF16 activations, got F16")
        if fp8 and x.dtype not in (torch.float32, torch.bfloat16):
            raise ValueError(f"nn.Linear: F8E4M3 weight needs F32/BF16/F16 activations, got {x.dtype}")
        w16 = (not quantized) and x.dtype == torch.float32 and self.W.dtype in (torch.bfloat16, torch.float16)
        if not quantized and not fp8 and not w16 and x.dtype != self.W.dtype:
            raise ValueError(f"nn.Linear: x dtype {x.dtype} != W dtype {self.W.dtype} — cast at the boundary, not inside the layer")
        flat = x.reshape(-1, self.in_features).contiguous()
        bias_done = False
        if fp8:
            y = ops.MatMulF8Block(flat, self.W, self.WBlockScale, self.WBlock[0], self.WBlock[1])
        elif quantized:
            y = ops.MatMulQ(flat, self.W)
        elif w16:
            y = flat @ self.W.float().t()          # the 16-bit weight widened exactly, F32 arithmetic (ops.MatMulW16)
        elif self.B is not None and self.W.dtype == torch.bfloat16:
            # one rounding for x W^T + b (nn/linear.go:312-322): F32 product, F32 bias add, then BF16
            y = (torch.mm(flat, self.W.t(), out_dtype=torch.float32) + self.B.float()).to(torch.bfloat16)
            bias_done = True
        else:
            y = flat @ self.W.t()
        if self.B is not None and not bias_done:
            y = y + self.B
        return y.reshape(*x.shape[:-1], self.out_features)

    def _forward_int4(self, x: torch.Tensor) -> torch.Tensor:
        w = self.W4
        if x.device != w.codes.device:
            raise ValueError(f"nn.Linear: x on {x.device} but the 4-bit weight on {w.codes.device}")
        if x.dim() < 1 or x.shape[-1] != self.in_features:
            raise ValueError(f"nn.Linear: last dim of x ({x.shape[-1] if x.dim() else 0}) != in_features ({self.in_features})")
        flat = x.reshape(-1, self.in_features)
        inp = flat.float() if (self.B is not None and x.dtype == torch.bfloat16) else flat   # bias added before the one rounding
        y = ops.MatMulInt4(inp, w)
        if self.B is not None:
            y = (y + self.B.to(y.dtype)).to(x.dtype)
        return y.reshape(*x.shape[:-1], self.out_features)


def _router_is_faster(T: int, E: int, K: int, f32: bool) -> bool:
    """Whether ops.RouterLogits takes less time than the library's f32 matmul does, with its pass over bf16 tokens to f32 (us, the library / here, tokens x experts x K).
    One token is the library's matrix-vector product: f32 1 x 64 x 2048 7.5 / 5.7, 1 x 256 x 1024 6.7 / 5.8, but 1 x 256 x 2048 5.2 / 6.1, 1 x 64 x 4096 7.8 / 9.3, 1 x 64 x 512
    3.6 / 6.0; bf16 1 x 256 x 4096 8.0 / 7.6, but 1 x 256 x 7168 9.2 / 11.4.  Short rows leave the tensor cores little to do beside the launch: f32 16 x 256 x 256 3.9 / 5.2, 512 x 256 x 768
    15.6 / 20.3, bf16 4096 x 40 x 256 13.2 / 25.0.  Few experts leave most of a tile of 64 of them empty: f32 1500 x 8 x 1280 19.7 / 22.6, bf16 4096 x 4 x 512
    19.8 / 26.0, 8192 x 8 x 1280 53 / 56.  F32 tokens cost six products to a weight where the library has one multiply-add: past 2^18 places in the tiles 3000 x 200 x 1536
    69 / 80 (4096 x 64 x 4096 1.5 times as fast here)."""
    wide, narrow = -(-T // 64) * -(-E // 64), -(-T // 16) * -(-E // 32)
    short = narrow * K <= 1 << 17  # (tiles of 16 x 32 even so: router.cu)
    if f32:
        if T == 1:
            return 1024 <= K < 1280 or (E <= 64 and 2048 <= K <= 3072)
        if K < 1024:
            return 16 < T <= 1024 and short and wide * 4096 <= 192 * K
        return wide <= 64 and (E > 16 or K >= 2048 or T <= 1024)
    if T == 1:
        return K <= 3072 or (K <= 5120 and E * K <= 1 << 20)
    if K < 512:
        return short and T <= 2000
    return E > 32 or K >= 2048 or T <= (4 * K if K < 1024 else 6 * K if E <= 16 else T)


@dataclass
class SparseMoE:
    """Routed gated-MLP block (nn/moe.go:27-60).  `GateUp` (E, 2 I, H) holds every expert's gate rows then up rows,
    `Down` (E, H, I); both dense tensors at the activation dtype or ops.QTensor (then activations are F32).
    Block-scaled FP8 experts carry `GateUpScale` / `DownScale` with `Block`.  `GateUpQ4` / `DownQ4` are per-expert 4-bit
    weights instead.  `Router`, when set, maps the (T, E) F32 router logits to an ops.MoERouting (the group-limited and
    sigmoid-with-bias routers); otherwise softmax + top-k."""
    Gate: Linear
    GateUp: Union[torch.Tensor, ops.QTensor, None] = None
    Down: Union[torch.Tensor, ops.QTensor, None] = None
    TopK: int = 1
    NormTopK: bool = False
    Gelu: bool = False
    RouterF32: bool = False
    Router: Optional[Callable[[torch.Tensor], ops.MoERouting]] = None
    GateUpQ4: Optional[Sequence[ops.Int4]] = None
    DownQ4: Optional[Sequence[ops.Int4]] = None
    GateUpScale: Optional[torch.Tensor] = None
    DownScale: Optional[torch.Tensor] = None
    Block: Tuple[int, int] = (0, 0)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        H = self.Gate.in_features
        if x.shape[-1] != H:
            raise ValueError(f"nn.SparseMoE: last dim {x.shape[-1]} != hidden {H}")
        flat = x.contiguous().reshape(-1, H)
        logits = self._logits_here(flat)
        if logits is not None:
            route = self._choose(logits)
        else:
            route = self.route(flat.float() if (self.RouterF32 and flat.dtype != torch.float32) else flat)
        if self.GateUpQ4 is not None:
            return ops.MoEInt4(flat, self.GateUpQ4, self.DownQ4, route, self.TopK, self.Gelu).reshape(x.shape)
        return self.run_experts(flat, route).reshape(x.shape)

    def route(self, gate_in: torch.Tensor) -> ops.MoERouting:
        return self._choose(self.Gate.forward(gate_in).float())

    def _choose(self, logits: torch.Tensor) -> ops.MoERouting:
        if self.Router is not None:
            return self.Router(logits)
        return ops.MoERoute(torch.softmax(logits, -1), self.TopK, self.NormTopK)

    def _logits_here(self, x: torch.Tensor) -> Optional[torch.Tensor]:
        """The router's matmul as ops.RouterLogits: a plain F32 gate on rows that it takes as they are, of a size where it is the faster one, where nothing is to
        see the matmul or to take its place (a route or a gate's forward of the program's own, on the class or on the object; autograd in either direction, transforms and
        modes: host.cpp); else None."""
        g = self.Gate
        w = g.W
        if getattr(self.route, "__func__", None) is not _ROUTE or type(g) is not Linear or getattr(g.forward, "__func__", None) is not _LINEAR or g.B is not None or \
                g.W4 is not None or type(w) is not torch.Tensor or type(x) is not torch.Tensor or \
                not (x.dtype == torch.float32 or (self.RouterF32 and x.dtype == torch.bfloat16)) or tuple(w.shape) != (g.out_features, g.in_features) or \
                torch.is_autocast_enabled("cuda") or not _router_is_faster(x.shape[0], *w.shape, x.dtype == torch.float32):
            return None
        return ops._host.router_logits(x, w)

    def run_experts(self, flat: torch.Tensor, route: ops.MoERouting) -> torch.Tensor:
        gu, dn = self.GateUp, self.Down
        quantized = isinstance(gu, ops.QTensor)
        if quantized and flat.dtype != torch.float32:
            raise ValueError(f"nn.SparseMoE: quantized experts ({ops.GGUF_NAMES[gu.ggml_type]}) need F32 activations, got {flat.dtype}")
        if quantized:
            gemm = lambda a, w, tw: ops.MoEGemmQ(a, w, route, tw, self.TopK)
        elif gu.dtype == torch.float8_e4m3fn:
            scale = {id(gu): self.GateUpScale, id(dn): self.DownScale}
            gemm = lambda a, w, tw: ops.MoEGemmF8Block(a, w, scale[id(w)], self.Block[0], self.Block[1], route, tw, self.TopK)
        else:
            gemm = lambda a, w, tw: ops.MoEGemm(a, w, route, tw, self.TopK)
        h = gemm(flat, gu, None)                          # (M, 2 I)
        pair = gemm(ops.MoEGateMul(h, self.Gelu), dn, route.weights)   # (M, H), routing-weighted
        return ops.MoECombine(pair, self.TopK)            # (T, H)


_LINEAR, _ROUTE = Linear.forward, SparseMoE.route
