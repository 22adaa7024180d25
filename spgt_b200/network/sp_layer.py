"""Sp_GalerkinAttention / Sp_EncoderLayer / Sp_SpectralConv2D: same constructors, parameter names and forward
signatures as the reference's network/sp_layer.py.  `forward` is the inference path, every step on the sm_100a kernels;
`forward_train` is the differentiable path the training loop uses (the reference's own op sequence: this library's
attention / projection / data-movement ops with their backward kernels, library ops for the rest).

Dropout: the reference calls F.dropout without `training=`, which keeps it active under model.eval()
(network/sp_layer.py:76,133).  These modules treat every drop rate as 0; use rates of 0 in the reference when
comparing outputs.
"""
import math

import torch
from torch import Tensor

from .. import ops
from .layer import FeedForward, _KernelWeights, _act, _dense, _linear_kn, _linear_tc


class Sp_GalerkinAttention(_KernelWeights):
    def __init__(self, dim_hidden, num_head, dim_position, norm_eps, attn_droprate, fc_droprate, xavier, diagonal,
                 symmetric) -> None:
        super().__init__()
        assert dim_hidden % 128 == 0 and dim_hidden // num_head == 32
        dim_head = dim_hidden // num_head
        self.dim_hidden, self.num_head, self.dim_head, self.dim_position = dim_hidden, num_head, dim_head, dim_position
        self.norm_eps, self.attn_droprate, self.fc_droprate = norm_eps, attn_droprate, fc_droprate
        P, E = torch.nn.Parameter, torch.empty
        self.weight_Q, self.weight_K, self.weight_V = (P(E([dim_hidden, dim_hidden])) for _ in range(3))
        self.bias_Q, self.bias_K, self.bias_V = (P(E([dim_hidden])) for _ in range(3))
        self.ln_weight_K, self.ln_weight_V = (P(E([num_head, dim_head])) for _ in range(2))
        self.ln_bias_K, self.ln_bias_V = (P(E([num_head, dim_head])) for _ in range(2))
        self.fc_layer = torch.nn.Linear(dim_hidden + dim_position * num_head, dim_hidden)
        self._reset_parameters(xavier, diagonal, symmetric)

    def _reset_parameters(self, xavier, diagonal, symmetric):
        # same initialisation as the reference (network/sp_layer.py:39-50)
        for weight in [self.weight_Q, self.weight_K, self.weight_V]:
            torch.nn.init.xavier_uniform_(weight, gain=xavier)
            if diagonal > 0:
                weight.data += diagonal * torch.diag(torch.ones(weight.size(-1)))
            if symmetric:
                weight.data += weight.data.T
        for bias in [self.bias_Q, self.bias_K, self.bias_V]:
            torch.nn.init.constant_(bias, 0)
        for lnw, lnb in zip([self.ln_weight_K, self.ln_weight_V], [self.ln_bias_K, self.ln_bias_V]):
            torch.nn.init.ones_(lnw)
            torch.nn.init.zeros_(lnb)

    def qkv_weight(self):
        return self._cached('wqkv', lambda: ops.TcWeight(
            torch.cat([self.weight_Q.detach(), self.weight_K.detach(), self.weight_V.detach()], dim=1).contiguous()))

    def fc_weight(self):
        return self._cached('fc', lambda: _linear_tc(self.fc_layer.weight))

    @property
    def fusable(self) -> bool:
        """Whether the fused layer kernels cover these widths."""
        return self.dim_hidden == 128 and self.num_head == 4 and self.dim_head == 32 and self.dim_position == 2

    def fill_native(self, w, ptr, images=None) -> None:
        """Device pointers of this layer's weights into a spgt_encoder_weights; `ptr` keeps what it is given alive."""
        if images is None:
            images = self._cached('images', lambda: ops.EncoderImages(_dense(self.weight_K), _dense(self.weight_V)))
        w.wkv, w.wq = ptr(images), ptr(_dense(self.weight_Q))
        w.wfc, w.bfc = ptr(_dense(self.fc_layer.weight)), ptr(self.fc_layer.bias.detach())
        w.bq, w.bk, w.bv = (ptr(b.detach()) for b in (self.bias_Q, self.bias_K, self.bias_V))
        w.lnwk, w.lnbk, w.lnwv, w.lnbv = (ptr(t.detach()) for t in (self.ln_weight_K, self.ln_bias_K, self.ln_weight_V, self.ln_bias_V))

    def forward(self, Q: Tensor, K: Tensor, V: Tensor, position: Tensor, residual: Tensor = None) -> Tensor:
        """Q,K,V [N,S,D], position [N,S,d_pos] -> [N,S,D] (+ residual, fused into the output projection).
        When Q, K and V are the same tensor (self-attention) all three projections run in one launch."""
        d = lambda t: t.detach()
        H, dh, dp = self.num_head, self.dim_head, self.dim_position
        if (Q is K and K is V and self.fusable and (residual is None or residual is Q)
                and ops.encoder_fused_pays(Q.shape[0], Q.shape[1], ffn=False)):
            plan = self._cached('native', lambda: ops.EncoderPlan(self.fill_native))
            return ops.encoder_layer(plan, Q, position, self.norm_eps, None, ffn=False, residual=residual is not None)
        if Q is K and K is V and self.dim_hidden == 128:
            q, k, v = ops.projpos_qkv_tc(
                Q, self.qkv_weight(), d(self.bias_Q), d(self.bias_K), d(self.bias_V), d(self.ln_weight_K), d(self.ln_bias_K),
                d(self.ln_weight_V), d(self.ln_bias_V), self.norm_eps, position, H, dh, dp)
        elif Q is K and K is V:
            q, k, v = ops.projpos_qkv(
                Q, d(self.weight_Q), d(self.bias_Q), d(self.weight_K), d(self.bias_K), d(self.weight_V), d(self.bias_V),
                d(self.ln_weight_K), d(self.ln_bias_K), d(self.ln_weight_V), d(self.ln_bias_V), self.norm_eps, position,
                H, dh, dp)
        else:
            q = ops.projpos(Q, d(self.weight_Q), d(self.bias_Q), position, H, dh, dp)
            k = ops.projpos_lnorm(K, d(self.weight_K), d(self.bias_K), d(self.ln_weight_K), d(self.ln_bias_K), position,
                                  self.norm_eps, H, dh, dp)
            v = ops.projpos_lnorm(V, d(self.weight_V), d(self.bias_V), d(self.ln_weight_V), d(self.ln_bias_V), position,
                                  self.norm_eps, H, dh, dp)
        X = ops.galerkin_attention(q, k, v, merged_heads=True)          # [N, S, H*(d_pos+d_head)]
        return ops.linear_tc(X, self.fc_weight(), d(self.fc_layer.bias), None, residual)


def _attention_forward_train(self, Q: Tensor, K: Tensor, V: Tensor, position: Tensor) -> Tensor:
    """Sp_GalerkinAttention.forward of the reference (network/sp_layer.py:52-78, drop rates 0) on the differentiable ops."""
    from ..extension.bind.galerkin_attention import (multihead_galerkin_attention_cccr_cuda,
                                                     multihead_projection_layernorm_with_position_rrc_cuda,
                                                     multihead_projection_with_position_rrc_cuda)
    H, dh, dp = self.num_head, self.dim_head, self.dim_position
    N, S, _ = Q.shape
    q = multihead_projection_with_position_rrc_cuda(Q, self.weight_Q, self.bias_Q, position, H, dh, dp)
    k = multihead_projection_layernorm_with_position_rrc_cuda(K, self.weight_K, self.bias_K, self.ln_weight_K, self.ln_bias_K,
                                                             position, self.norm_eps, H, dh, dp)
    v = multihead_projection_layernorm_with_position_rrc_cuda(V, self.weight_V, self.bias_V, self.ln_weight_V, self.ln_bias_V,
                                                             position, self.norm_eps, H, dh, dp)
    X = multihead_galerkin_attention_cccr_cuda(q, k, v)                  # [N, H, S, d_pos + d_head]
    X = X.transpose(1, 2).contiguous().view(N, S, H * (dp + dh))
    return self.fc_layer(X)


Sp_GalerkinAttention.forward_train = _attention_forward_train


def _encoder_layer_by_ops(x: Tensor, position: Tensor, eps: float, params) -> Tensor:
    """The encoder layer (width 128, 4 heads, 2 position values, ReLU) on the single differentiable ops."""
    from ..extension.bind.galerkin_attention import (multihead_galerkin_attention_cccr_cuda,
                                                     multihead_projection_layernorm_with_position_rrc_cuda,
                                                     multihead_projection_with_position_rrc_cuda)
    wq, bq, wk, bk, wv, bv, lnwk, lnbk, lnwv, lnbv, wfc, bfc, w1, b1, w2, b2 = params
    linear = torch.nn.functional.linear
    q = multihead_projection_with_position_rrc_cuda(x, wq, bq, position, 4, 32, 2)
    k = multihead_projection_layernorm_with_position_rrc_cuda(x, wk, bk, lnwk, lnbk, position, eps, 4, 32, 2)
    v = multihead_projection_layernorm_with_position_rrc_cuda(x, wv, bv, lnwv, lnbv, position, eps, 4, 32, 2)
    att = multihead_galerkin_attention_cccr_cuda(q, k, v).transpose(1, 2).reshape(x.shape[0], x.shape[1], 136)
    x = x + linear(att, wfc, bfc)
    return x + linear(torch.relu(linear(x, w1, b1)), w2, b2)


def _as_read(params) -> list:
    """The parameters as the kernels read them: themselves where they are row-major and 16-byte aligned."""
    return [p if p.is_contiguous() and p.data_ptr() % 16 == 0 else _dense(p) for p in params]


class _EncoderLayerFunction(torch.autograd.Function):
    """X + attention(X), then + ffn(.): projections and attention in one native call, their backward and all weight gradients in
    another; the dense layers' products along the layer are plain fp32, whose last bits decide what passes the ReLU.  A backward
    pass that is to be differentiated again (create_graph) runs on the single ops, whose gradients carry a graph."""

    @staticmethod
    def forward(ctx, x, position, eps, *params):
        ctx.eps, inputs = eps, (x, position, *params)
        x, params = x.contiguous(), _as_read(params)
        att, saved = ops.encoder_train_forward(x, position.contiguous(), eps, params)
        linear = torch.nn.functional.linear
        x1 = x + linear(att, params[10], params[11])
        h = torch.relu(linear(x1, params[12], params[13]))
        ctx.save_for_backward(att, x1, h, saved, *inputs)
        return x1 + linear(h, params[14], params[15])

    @staticmethod
    def backward(ctx, grad_out):
        att, x1, h, saved, x, position, *params = ctx.saved_tensors
        if torch.is_grad_enabled():
            wanted = [t for t, need in zip((x, *params), (ctx.needs_input_grad[0], *ctx.needs_input_grad[3:])) if need]
            grads = iter(torch.autograd.grad(_encoder_layer_by_ops(x, position, ctx.eps, params), wanted, grad_out, create_graph=True))
            return tuple(next(grads) if need else None for need in ctx.needs_input_grad)
        dx, grads = ops.encoder_train_backward(x.contiguous(), att, x1, h, ctx.eps, _as_read(params), saved, _dense(grad_out))
        return (dx, None, None, *grads)


class Sp_EncoderLayer(_KernelWeights):
    def __init__(self, dim_hidden, num_head, dim_position, norm_eps, attn_droprate, fc_droprate, xavier, diagonal,
                 symmetric, ffn_dim_hidden, ffn_droprate, ffn_activation) -> None:
        super().__init__()
        self.attention_layer = Sp_GalerkinAttention(
            dim_hidden, num_head, dim_position, norm_eps, attn_droprate, fc_droprate, xavier, diagonal, symmetric)
        self.ffn_layer = FeedForward(dim_hidden, dim_hidden, ffn_dim_hidden, ffn_droprate, ffn_activation)

    def fill_native(self, w, ptr) -> None:
        a, f = self.attention_layer, self.ffn_layer
        images = self._cached('images', lambda: ops.EncoderImages(*(_dense(t) for t in (a.weight_K, a.weight_V, f.layer1.weight, f.layer2.weight))))
        a.fill_native(w, ptr, images)
        w.w1, w.w2 = images.data_ptr() + images.stride, images.data_ptr() + 2 * images.stride
        w.b1, w.b2 = ptr(f.layer1.bias.detach()), ptr(f.layer2.bias.detach())

    def forward(self, X: Tensor, position: Tensor) -> Tensor:
        """X [N,S,D], position [N,S,d_pos] -> X + attention(X) then + ffn(.)  (network/sp_layer.py:94-104)."""
        f = self.ffn_layer
        if self.fusable and not self._watch.observed(self) and ops.encoder_fused_pays(X.shape[0], X.shape[1]):
            plan = self._cached('native', lambda: ops.EncoderPlan(self.fill_native))
            return ops.encoder_layer(plan, X, position, self.attention_layer.norm_eps, f.activation)
        X = self.attention_layer(X, X, X, position, residual=X)
        return f(X, residual=X)

    @property
    def fusable(self) -> bool:
        f = self.ffn_layer
        return (type(self.attention_layer) is Sp_GalerkinAttention and type(f) is FeedForward and f.fused
                and self.attention_layer.fusable and type(f.layer1) is torch.nn.Linear and type(f.layer2) is torch.nn.Linear
                and f.layer1.in_features == 128 and f.layer1.out_features == 256
                and f.layer2.out_features == 128)

    def trains_fused(self) -> bool:
        """Whether the fused training layer stands for this one: its widths and activation, the modules' own linear layers, nothing
        that watches or alters their calls or the gradients through them."""
        a, f = self.attention_layer, self.ffn_layer
        if not self.fusable or f.activation != 'relu':
            return False
        linears = (a.fc_layer, f.layer1, f.layer2)
        return (all(type(l) is torch.nn.Linear and l.bias is not None for l in linears)
                and all(b is not None for b in (a.bias_Q, a.bias_K, a.bias_V))
                and not self._watch.observed(self) and not self._watch.backward_observed(*linears))

    def forward_train(self, X: Tensor, position: Tensor) -> Tensor:
        a, f = self.attention_layer, self.ffn_layer
        if X.is_cuda and X.dim() == 3 and X.dtype == torch.float32 and not torch.is_autocast_enabled() and self.trains_fused():
            return _EncoderLayerFunction.apply(
                X, position, a.norm_eps, a.weight_Q, a.bias_Q, a.weight_K, a.bias_K, a.weight_V, a.bias_V, a.ln_weight_K, a.ln_bias_K,
                a.ln_weight_V, a.ln_bias_V, a.fc_layer.weight, a.fc_layer.bias, f.layer1.weight, f.layer1.bias, f.layer2.weight, f.layer2.bias)
        X = X + self.attention_layer.forward_train(X, X, X, position)
        return X + self.ffn_layer.forward_train(X)


class Sp_SpectralConv2D(_KernelWeights):
    """structure='fused' (default): one mode-truncated DFT pipeline (spgt_spectral_conv2d_fwd).
    structure='reference': the reference's own op sequence (network/sp_layer.py:125-156): batched_transpose ->
    torch.fft.rfft2 -> transpose_gather_dual -> complex matmul -> transpose_scatter_dual -> torch.fft.irfft2 ->
    batched_transpose, which exercises the data-movement ops in context."""

    def __init__(self, in_dim, out_dim, mode, droprate, activation, structure: str = 'fused') -> None:
        super().__init__()
        self.in_dim, self.out_dim, self.mode, self.droprate = in_dim, out_dim, mode, droprate
        self.activation = activation
        self.structure = structure
        self.residual_layer = torch.nn.Linear(in_dim, out_dim)
        self.fourier_weight = torch.nn.ParameterList([
            torch.nn.Parameter(torch.empty([mode, mode, in_dim, out_dim, 2])) for _ in range(2)])
        for param in self.fourier_weight:
            torch.nn.init.xavier_normal_(param, gain=1.0 / (in_dim * out_dim) * math.sqrt(in_dim + out_dim))

    def residual_weight(self):
        return self._cached('wr', lambda: _linear_kn(self.residual_layer.weight))

    def fill_native(self, w, ptr) -> None:
        w.wr, w.br = ptr(self.residual_weight()), ptr(self.residual_layer.bias.detach())
        w.fw0, w.fw1 = (ptr(p.detach()) for p in self.fourier_weight)

    def forward(self, X: Tensor) -> Tensor:
        N, r, _, in_dim = X.shape
        m, out_dim = self.mode, self.out_dim
        wr = self.residual_weight()
        br = self.residual_layer.bias.detach()
        fw0, fw1 = self.fourier_weight[0].detach(), self.fourier_weight[1].detach()
        if self.structure == 'fused':
            return ops.spectral_conv2d(X, wr, br, fw0, fw1, m, self.activation)
        from ..extension.bind.datamove import batched_transpose, transpose_gather_dual, transpose_scatter_dual
        Xt = batched_transpose(X, [N], [r, r], [in_dim])
        X_ft = torch.fft.rfft2(Xt, s=(r, r), norm='ortho').contiguous()
        a, b = transpose_gather_dual(X_ft, [N, in_dim], r, r // 2 + 1, m, m, 0, 0, r - m, 0)
        a = a @ torch.view_as_complex(fw0)
        b = b @ torch.view_as_complex(fw1)
        Out_ft = transpose_scatter_dual(a.contiguous(), b.contiguous(), [N, out_dim], r, r // 2 + 1, m, m, 0, 0, r - m, 0)
        Y = torch.fft.irfft2(Out_ft, s=(r, r), norm='ortho').contiguous()
        Y = batched_transpose(Y, [N], [out_dim], [r, r])
        res = ops.linear(X, wr, br, out_dim, None, Y)             # X @ Wr + br + Y
        return torch.nn.functional.silu(res) if self.activation == 'silu' else torch.relu(res)

    def forward_train(self, X: Tensor) -> Tensor:
        """Differentiable path: the reference's op sequence (network/sp_layer.py:125-156, drop rate 0)."""
        from ..extension.bind.datamove import batched_transpose, transpose_gather_dual, transpose_scatter_dual
        N, r, _, in_dim = X.shape
        m, out_dim = self.mode, self.out_dim
        res = self.residual_layer(X)
        Xt = batched_transpose(X.contiguous(), [N], [r, r], [in_dim])
        X_ft = torch.fft.rfft2(Xt, s=(r, r), norm='ortho').contiguous()
        a, b = transpose_gather_dual(X_ft, [N, in_dim], r, r // 2 + 1, m, m, 0, 0, r - m, 0)
        a = a @ torch.view_as_complex(self.fourier_weight[0])
        b = b @ torch.view_as_complex(self.fourier_weight[1])
        Out_ft = transpose_scatter_dual(a.contiguous(), b.contiguous(), [N, out_dim], r, r // 2 + 1, m, m, 0, 0, r - m, 0)
        Y = torch.fft.irfft2(Out_ft, s=(r, r), norm='ortho').contiguous()
        Y = batched_transpose(Y, [N], [out_dim], [r, r])
        return _act(self.activation)(Y + res)
