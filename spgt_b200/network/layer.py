"""Shared layers of the Darcy model with the reference's parameter names (network/layer.py).

Each module keeps ordinary torch Parameters (so a reference state_dict loads unchanged) and a cache of the same
weights re-laid-out for the kernels ([K, N] row-major, column count padded to a multiple of 4).  `forward` is the
inference path on the fused kernels; `forward_train` is the differentiable path of the training loop, which - like
the reference's own SpGT training - runs the convolutions, interpolations, dense layers and FFTs as library ops
under torch autograd and the attention / projection / data-movement steps on this library's ops and their backward
kernels.
"""
import torch
from torch import Tensor
from torch.nn.modules import module as _hooks

from .. import ops


class ParameterWatch:
    """Tells when a module is not as it was seen before: tag() differs after a parameter has been written to (an optimizer step
    bumps the version counters), moved, or replaced, a submodule has been exchanged, or an option that kernels are chosen by
    has been set.  The tree is walked once, not on every call (Module.parameters() takes longer than the launch it would guard)."""
    OPTIONS = ('activation', 'norm_eps', 'mode', 'structure', 'fused')

    def __init__(self):
        # one tuple, replaced whole: several threads may share a module.  It holds neither the module nor its __dict__, which would
        # be a cycle that keeps the module's memory until a garbage collection
        self._tree = None

    def _walk(self, module: torch.nn.Module) -> tuple:
        modules = list(module.modules())
        return ([(d, len(d)) for m in modules for d in (m._modules, m._parameters)],
                [(m._modules, k, c) for m in modules for k, c in m._modules.items()],
                [(m._parameters, k) for m in modules for k in m._parameters],
                [(m.__dict__, k) for m in modules[1:] for k in self.OPTIONS if k in m.__dict__],
                [m.__dict__ for m in modules[1:]])

    def _seen(self, module: torch.nn.Module) -> tuple:
        tree = self._tree
        try:
            if tree is not None and not any(len(d) != n for d, n in tree[0]) and not any(d[k] is not c for d, k, c in tree[1]):
                return tree
        except KeyError:                                  # a submodule under another name: as many entries as before
            pass
        tree = self._tree = self._walk(module)
        return tree

    def tag(self, module: torch.nn.Module) -> tuple:
        tree = self._seen(module)
        try:
            params = [d[k] for d, k in tree[2]]
            values = [p._version for p in params] + [p.data_ptr() for p in params]
        except (KeyError, AttributeError):                # renamed (pruning, spectral normalisation), or None in place of a bias
            tree = self._tree = self._walk(module)
            params = [d[k] for d, k in tree[2]]
            values = [(0, 0) if p is None else (p._version, p.data_ptr()) for p in params]
        return tuple(values + [d.get(k) for d, k in tree[3]] + [module.__dict__.get(k) for k in self.OPTIONS])

    def observed(self, module: torch.nn.Module) -> bool:
        """Whether a submodule's call can be told from a call of its kernels: forward hooks, or a forward of its own."""
        if _hooks._global_forward_hooks or _hooks._global_forward_pre_hooks:
            return True
        return any(d['_forward_hooks'] or d['_forward_pre_hooks'] or 'forward' in d for d in self._seen(module)[4])

    def backward_observed(self, *called: torch.nn.Module) -> bool:
        """Whether hooks wait for the gradients that pass the modules `called`: they fire, and may replace the gradients, only where
        the modules themselves are called."""
        if _hooks._global_backward_hooks or _hooks._global_backward_pre_hooks:
            return True
        return any(m._backward_hooks or m._backward_pre_hooks for m in called)

    def hold(self, module: torch.nn.Module) -> list:
        """Aliases of the parameters' storages: while they are kept, no other tensor can come to lie at these addresses."""
        return [d[k].detach() for d, k in self._seen(module)[2] if d.get(k) is not None]

    def __deepcopy__(self, memo):
        return ParameterWatch()


class _KernelWeights(torch.nn.Module):
    """Caches derived weight layouts; the cache is dropped whenever parameters are (re)loaded or moved."""

    def __init__(self):
        super().__init__()
        self._kw = {}
        self._watch = ParameterWatch()
        self.register_load_state_dict_post_hook(lambda module, incompatible: module._kw.clear())

    def _apply(self, fn, *args, **kwargs):
        self._kw.clear()
        return super()._apply(fn, *args, **kwargs)

    def __getstate__(self):
        return {**self.__dict__, '_kw': {}}      # derived layouts (device pointers among them) are not copied with the module

    def _cached(self, key, make):
        """Derived layout of the module's weights, rebuilt when a parameter is not the one it was made from."""
        tag = self._watch.tag(self)
        hit = self._kw.get(key)
        if hit is None or hit[0] != tag:
            with torch.no_grad():
                hit = (tag, make(), self._watch.hold(self))
            self._kw[key] = hit
        return hit[1]


def _dense(weight: Tensor) -> Tensor:
    """A weight that a kernel reads as it is: row-major and 16-byte aligned, copied only where it is not."""
    w = weight.detach().contiguous()
    return w if w.data_ptr() % 16 == 0 else w.clone()


def _linear_kn(weight: Tensor) -> Tensor:
    """torch Linear weight [out, in] -> [in, out4] row-major."""
    return ops.pad_cols(weight.detach().t().contiguous())


def _conv_kn(weight: Tensor) -> Tensor:
    """Conv2d weight [Cout, Cin, 3, 3] -> [(ky*3+kx)*Cin + ci, Cout4] row-major."""
    cout, cin = weight.shape[:2]
    return ops.pad_cols(weight.detach().permute(2, 3, 1, 0).reshape(9 * cin, cout).contiguous())


def _linear_tc(weight: Tensor) -> 'ops.TcWeight':
    """torch Linear weight [out, in] prepared for the tcgen05 GEMM."""
    return ops.TcWeight(_dense(weight), transposed=True)


def _conv_tc(weight: Tensor, bias: Tensor, cin_pad: int, cout_pad: int, tiles: bool = True):
    """Conv2d weight [Cout, Cin, 3, 3] (+ bias) prepared for the convolution kernel (`tiles`; up to 128 output channels) or the implicit
    GEMM, with input / output channels zero-padded to cin_pad / cout_pad (padded outputs come out as act(0))."""
    if tiles and cout_pad <= 128:
        return ops.ConvWeight.padded(weight.detach().contiguous(), bias.detach().contiguous(), cin_pad, cout_pad)
    cout, cin = weight.shape[:2]
    w = torch.zeros(cout_pad, cin_pad, 3, 3, device=weight.device, dtype=weight.dtype)
    w[:cout, :cin] = weight.detach()
    b = torch.zeros(cout_pad, device=weight.device, dtype=weight.dtype)
    b[:cout] = bias.detach()
    return ops.TcWeight(w.permute(2, 3, 1, 0).reshape(9 * cin_pad, cout_pad).contiguous()), b


class ConvResBlock2D(_KernelWeights):
    """conv3x3(pad 1) -> [dropout, rate treated as 0] -> activation; NHWC in and out.
    Reference: network/layer.py:7-24 (NCHW there; the kernels keep channels last throughout)."""

    def __init__(self, in_dim, out_dim, kernel_size, padding, droprate, activation) -> None:
        super().__init__()
        assert kernel_size == 3 and padding == 1
        self.droprate = droprate
        self.activation = activation
        self.conv_layer = torch.nn.Conv2d(in_dim, out_dim, kernel_size=kernel_size, padding=padding)

    def kernel_weight(self):
        return self._cached('w', lambda: _conv_kn(self.conv_layer.weight))

    def forward_train(self, X: Tensor) -> Tensor:
        """NCHW in and out, differentiable (network/layer.py:16-24 with drop rate 0)."""
        return _act(self.activation)(self.conv_layer(X))

    def forward_nhwc(self, X: Tensor, cin_off: int, out: Tensor, cout_off: int, act=None) -> Tensor:
        """Generic path (any even channel counts / offsets): warp-MMA implicit GEMM."""
        w = self.conv_layer.weight
        return ops.conv3x3(X, cin_off, w.shape[1], self.kernel_weight(), self.conv_layer.bias.detach(), out, cout_off,
                           w.shape[0], self.activation if act is None else act)

    def tc_weight(self, cin_pad: int, cout_pad: int, tiles: bool = True):
        return self._cached(('tc', cin_pad, cout_pad, tiles), lambda: _conv_tc(self.conv_layer.weight, self.conv_layer.bias, cin_pad, cout_pad, tiles))

    def forward_tc(self, X: Tensor, cin_pad: int, cout_pad: int, act=None) -> Tensor:
        """tcgen05 path: X [N,H,W,cin_pad] (channels beyond in_dim must be finite; their weights are zero) ->
        new tensor [N,H,W,cout_pad] whose channels beyond out_dim hold act(0)."""
        wt, b = self.tc_weight(cin_pad, cout_pad, ops.conv3x3_tiles_pay(*X.shape[:3], X.device))
        out = torch.empty(*X.shape[:3], cout_pad, device=X.device, dtype=X.dtype)
        return ops.conv3x3_tc(X, 0, cin_pad, wt, b, out, 0, cout_pad, self.activation if act is None else act)


def _act(name):
    """The reference selects SiLU for 'silu' and ReLU for any other string (network/layer.py:14,163)."""
    return torch.nn.functional.silu if name == 'silu' else torch.relu


class FeedForward(_KernelWeights):
    """Linear -> activation -> Linear (dropout rate treated as 0).  Reference: network/layer.py:155-174."""

    def __init__(self, in_dim, out_dim, dim_hidden, droprate, activation) -> None:
        super().__init__()
        self.droprate = droprate
        self.activation = activation
        self.layer1 = torch.nn.Linear(in_dim, dim_hidden)
        self.layer2 = torch.nn.Linear(dim_hidden, out_dim)
        self.fused = True        # one kernel for both GEMMs when the shape is 128 -> 256 -> 128

    def tc_weights(self):
        return self._cached('w1', lambda: _linear_tc(self.layer1.weight)), self._cached('w2', lambda: _linear_tc(self.layer2.weight))

    def forward(self, X: Tensor, residual: Tensor = None) -> Tensor:
        """X [..., in_dim] -> [..., out_dim] (+ residual when given, fused into the second GEMM)."""
        w1, w2 = self.tc_weights()
        if self.fused and w1.K == 128 and w1.N == 256 and w2.N == 128:
            return ops.ffn_tc(X, w1, self.layer1.bias.detach(), w2, self.layer2.bias.detach(), self.activation, residual)
        h = ops.linear_tc(X, w1, self.layer1.bias.detach(), self.activation)
        return ops.linear_tc(h, w2, self.layer2.bias.detach(), None, residual)

    def forward_train(self, X: Tensor) -> Tensor:
        return self.layer2(_act(self.activation)(self.layer1(X)))
