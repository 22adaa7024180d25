"""Sp_EncoderMixer / Sp_DecoderRegressor / Sp_GalerkinTransformer2D: same constructors, parameter names
(state_dict keys) and forward signatures as the reference's network/sp_model.py.  Without gradients (eval, or
torch.no_grad) the forward runs on the fused inference kernels; in training mode with gradients enabled it runs the
differentiable path (`forward_train` of the modules)."""
import numpy as np
import torch
from torch import Tensor

from .. import ops
from .._lib import MAX_LAYERS, DarcyModel
from .layer import ConvResBlock2D, FeedForward, ParameterWatch, _KernelWeights, _linear_kn, _linear_tc
from .model import DownScaler2D, UpScaler2D
from .sp_layer import Sp_EncoderLayer, Sp_SpectralConv2D


class Sp_EncoderMixer(torch.nn.Module):
    def __init__(self, num_layer, dim_hidden, num_head, dim_position, norm_eps, attn_droprate, fc_droprate, xavier,
                 diagonal, symmetric, ffn_dim_hidden, ffn_droprate, ffn_activation) -> None:
        super().__init__()
        self.layers = torch.nn.ModuleList([
            Sp_EncoderLayer(dim_hidden, num_head, dim_position, norm_eps, attn_droprate, fc_droprate, xavier, diagonal,
                            symmetric, ffn_dim_hidden, ffn_droprate, ffn_activation) for _ in range(num_layer)])

    def forward(self, X: Tensor, position: Tensor) -> Tensor:
        N, r_attn, _, dim_hidden = X.shape
        X = X.view(N, r_attn * r_attn, dim_hidden)
        position = position.reshape(N, r_attn * r_attn, position.size(-1))
        for layer in self.layers:
            X = layer(X, position)
        return X.view(N, r_attn, r_attn, dim_hidden)

    def forward_train(self, X: Tensor, position: Tensor) -> Tensor:
        N, r_attn, _, dim_hidden = X.shape
        X = X.reshape(N, r_attn * r_attn, dim_hidden)
        position = position.reshape(N, r_attn * r_attn, position.size(-1)).contiguous()
        for layer in self.layers:
            X = layer.forward_train(X, position)
        return X.view(N, r_attn, r_attn, dim_hidden)


class Sp_DecoderRegressor(_KernelWeights):
    def __init__(self, num_layer, in_dim, out_dim, dim_position, dim_spatial_hidden, mode, droprate, activation) -> None:
        super().__init__()
        assert out_dim == 1, 'the fused decoder head produces the scalar Darcy target'
        self.in_dim, self.dim_position, self.activation = in_dim, dim_position, activation
        self.spatial_fc_layer = torch.nn.Linear(in_dim + dim_position, dim_spatial_hidden)
        self.layers = torch.nn.ModuleList([
            Sp_SpectralConv2D(dim_spatial_hidden, dim_spatial_hidden, mode, droprate, activation) for _ in range(num_layer)])
        dim_ffn_hidden = 2 * dim_position * dim_spatial_hidden
        self.ffn_layer = FeedForward(dim_spatial_hidden, out_dim, dim_ffn_hidden, droprate, activation)

    def head_weights(self):
        """(first weight as its kernel takes it, second weight [hidden]) of the decoder head."""
        f = self.ffn_layer
        make = _linear_tc if f.layer1.out_features == 128 else _linear_kn
        return self._cached('w1', lambda: make(f.layer1.weight)), self._cached('w2', lambda: f.layer2.weight.detach().reshape(-1).contiguous())

    def _spectral_and_head(self, X: Tensor, scale, shift, dirichlet, scale_map=None, shift_map=None) -> Tensor:
        for layer in self.layers:
            X = layer(X)
        f = self.ffn_layer
        w1, w2 = self.head_weights()
        b2 = self._cached('b2', lambda: float(f.layer2.bias.detach().reshape(-1)[0]))
        if f.layer1.out_features == 128:
            return ops.decoder_head_tc(X, w1, f.layer1.bias.detach(), w2, b2, scale, shift, dirichlet, self.activation,
                                       scale_map, shift_map)
        return ops.decoder_head(X, w1, f.layer1.bias.detach(), w2, b2, scale, shift, dirichlet, self.activation,
                                scale_map, shift_map)

    def forward(self, X: Tensor, grid: Tensor = None) -> Tensor:
        """X [N,r,r,in_dim], grid [N,r,r,d_pos] -> [N,r,r,1]  (network/sp_model.py:53-64)."""
        return self._spectral_and_head(self._fc_split(X, grid), 1.0, 0.0, False)

    def forward_train(self, X: Tensor, grid: Tensor) -> Tensor:
        """Differentiable path (network/sp_model.py:53-64)."""
        X = self.spatial_fc_layer(torch.concat([X, grid], dim=-1))
        for layer in self.layers:
            X = layer.forward_train(X)
        return self.ffn_layer.forward_train(X)

    def _fc_split(self, X, grid):
        """spatial_fc_layer(concat(X, grid)) = X @ Wx + grid @ Wg + b without materialising the concatenation."""
        wx, wg = self._split_fc()
        uw = ops.linear_tc(X, wx, None, None)
        return ops.upsample_grid(uw, grid, wg, self.spatial_fc_layer.bias.detach(), X.shape[1], X.shape[2])

    def _split_fc(self):
        w = self.spatial_fc_layer.weight
        wx = self._cached('wx', lambda: _linear_tc(w[:, :self.in_dim]))
        wg = self._cached('wg', lambda: w.detach()[:, self.in_dim:].t().contiguous())
        return wx, wg

    def forward_from_mid(self, U: Tensor, grid: Tensor, scale, shift, dirichlet, scale_map=None, shift_map=None) -> Tensor:
        """U [N,r_mid,r_mid,in_dim] is the up-scaler output BEFORE its last interpolation.  Interpolation and
        Linear are both linear maps, so Linear(concat(resize(U), grid)) = resize(U @ Wx) + grid @ Wg + b: the
        in_dim-channel full-resolution tensor is never formed."""
        wx, wg = self._split_fc()
        uw = ops.linear_tc(U, wx, None, None)
        X = ops.upsample_grid(uw, grid, wg, self.spatial_fc_layer.bias.detach(), grid.shape[1], grid.shape[2])
        return self._spectral_and_head(X, scale, shift, dirichlet, scale_map, shift_map)


def _normalizer_affine(normalizer, r: int, device):
    """(scale, shift, scale_map, shift_map) of inverse_transform(X) = X * (std + eps) + mean."""
    if normalizer is None:
        return 1.0, 0.0, None, None
    eps = float(getattr(normalizer, 'eps', 1.0e-5))
    mean = torch.as_tensor(np.asarray(normalizer.mean.cpu() if isinstance(normalizer.mean, torch.Tensor) else normalizer.mean),
                           dtype=torch.float32)
    std = torch.as_tensor(np.asarray(normalizer.std.cpu() if isinstance(normalizer.std, torch.Tensor) else normalizer.std),
                          dtype=torch.float32)
    if mean.numel() == 1 and std.numel() == 1:
        return float(std.reshape(-1)[0]) + eps, float(mean.reshape(-1)[0]), None, None
    scale_map = (std.reshape(-1) + eps).expand(r * r).contiguous().to(device) if std.numel() in (1, r * r) else None
    shift_map = mean.reshape(-1).expand(r * r).contiguous().to(device) if mean.numel() in (1, r * r) else None
    if scale_map is None or shift_map is None:
        raise ValueError('target normalizer statistics must be scalars or one value per grid node')
    return 1.0, 0.0, scale_map, shift_map


class Sp_GalerkinTransformer2D(torch.nn.Module):
    """Darcy Galerkin Transformer forward: down-scaler -> encoder layers -> up-scaler -> spectral regressor ->
    de-normalisation -> Dirichlet frame (network/sp_model.py:67-113).  cfg carries the keys of the reference's
    config (config/darcy_config.yaml) plus 'resolution_size' and 'target_normalizer'."""

    def __init__(self, cfg) -> None:
        super().__init__()
        self.droprate = cfg['drop_module']
        self.boundary_condition = cfg['boundary_condition']
        self.normalizer = cfg.get('target_normalizer')
        self.down_scaler = DownScaler2D(cfg['resolution_size'], cfg['dim_node'], cfg['dim_hidden'], cfg['drop_downscaler'],
                                        cfg['acti_downscaler'])
        self.encoder_mixer = Sp_EncoderMixer(
            cfg['num_encoder_layer'], cfg['dim_hidden'], cfg['num_head'], cfg['dim_position'], cfg['attn_norm_eps'],
            cfg['drop_encoder_attn'], cfg['drop_encoder_attn_fc'], cfg['attn_xavier'], cfg['attn_diagonal'],
            cfg['attn_symmetric'], cfg['dim_encoder_ffn'], cfg['drop_encoder_ffn'], cfg['acti_encoder_ffn'])
        self.up_scaler = UpScaler2D(cfg['resolution_size'], cfg['dim_hidden'], cfg['dim_hidden'], cfg['drop_upscaler'],
                                    cfg['acti_upscaler'])
        self.decoder_regressor = Sp_DecoderRegressor(
            cfg['num_decoder_layer'], cfg['dim_hidden'], cfg['dim_target'], cfg['dim_position'], cfg['dim_spatial_hidden'],
            cfg['num_frequence_mode'], cfg['drop_decoder_layer'], cfg['acti_decoder_layer'])
        self._affine = None
        self._plan, self._watch = None, ParameterWatch()

    def forward(self, X: Tensor, position: Tensor, grid: Tensor, taps: dict = None) -> Tensor:
        """X [N,r,r,1], position [N,r_attn,r_attn,2], grid [N,r,r,2] -> [N,r,r,1]; CUDA fp32 contiguous tensors.
        `taps`, when a dict, receives intermediate tensors (down-scaler output, each encoder layer, ...).
        In training mode with gradients enabled the differentiable path runs; otherwise the fused inference kernels."""
        if self.training and torch.is_grad_enabled():
            return self.forward_train(X, position, grid)
        with torch.no_grad():
            return self._forward_fused(X, position, grid, taps)

    def forward_train(self, X: Tensor, position: Tensor, grid: Tensor) -> Tensor:
        """The reference's forward (network/sp_model.py:91-113, every drop rate 0) on differentiable ops."""
        X = self.down_scaler.forward_train(X)
        X = self.encoder_mixer.forward_train(X, position)
        X = self.up_scaler.forward_train(X)
        X = self.decoder_regressor.forward_train(X, grid)
        r = X.shape[1]
        scale, shift, scale_map, shift_map = _normalizer_affine(self.normalizer, r, X.device)    # X * (std + eps) + mean
        X = X * (scale if scale_map is None else scale_map.view(1, r, r, 1)) + (shift if shift_map is None else shift_map.view(1, r, r, 1))
        if self.boundary_condition == 'dirichlet':
            X = torch.nn.functional.pad(X[:, 1:-1, 1:-1].contiguous(), (0, 0, 1, 1, 1, 1), 'constant', 0)
        return X

    def _forward_fused(self, X: Tensor, position: Tensor, grid: Tensor, taps: dict = None) -> Tensor:
        if ops.profiling() or self._watch.observed(self) or not self._native_shapes(X, position, grid):
            plan = None
        else:
            plan = self._native_plan(X)
        if plan is None:
            return self._forward_modules(X, position, grid, taps)
        return ops.darcy_forward(plan, X, position, grid, taps)

    def _native_shapes(self, X: Tensor, position: Tensor, grid: Tensor) -> bool:
        """Whether the inputs are one sample per coordinate set on the model's own grids, and not many samples of few nodes.  The modules
        also take a `grid` of other nodes (the regressor is evaluated there) or with more samples than X."""
        if type(self.down_scaler) is not DownScaler2D:
            return False
        (r, _), _, (ra, _) = self.down_scaler.resolution_size[:3]
        N = X.shape[0]
        return (tuple(X.shape) == (N, r, r, 1) and tuple(grid.shape) == (N, r, r, 2) and position.numel() == N * ra * ra * 2
                and position.shape[-1] == 2 and ops.encoder_fused_pays(N, ra * ra))

    def _native_plan(self, X: Tensor):
        """The model as the one-call forward takes it, rebuilt when the parameters, the grid or the device are not the ones it was
        made for; None for widths that forward does not cover."""
        if not (type(self.down_scaler) is DownScaler2D and type(self.up_scaler) is UpScaler2D):
            return None
        sizes = [tuple(map(tuple, m.resolution_size)) for m in (self.down_scaler, self.up_scaler)]
        tag = (X.shape[1], X.device, self.normalizer, self.boundary_condition, sizes, self._watch.tag(self))
        plan = self._plan                                    # (read once: another thread may replace it)
        if plan is None or plan[0] != tag:
            plan = self._plan = (tag, self._build_plan(X), self._watch.hold(self))
        return plan[1]

    def __getstate__(self):
        return {**self.__dict__, '_plan': None}              # device pointers are not copied with the module

    def _normalizer_terms(self, r: int, device):
        affine = self._affine
        if affine is None or affine[0] != (r, device, self.normalizer):
            affine = self._affine = ((r, device, self.normalizer), _normalizer_affine(self.normalizer, r, device))
        return affine[1]

    def _apply(self, fn, *args, **kwargs):
        self._plan = self._affine = None
        return super()._apply(fn, *args, **kwargs)

    def _build_plan(self, X: Tensor):
        r, down, up, dec = X.shape[1], self.down_scaler, self.up_scaler, self.decoder_regressor
        enc = list(self.encoder_mixer.layers)
        if not self._native_widths() or sum(down.dims) != 128 or max(len(enc), len(dec.layers)) > MAX_LAYERS:
            return None
        size = tuple(map(tuple, down.resolution_size))
        if size != tuple(map(tuple, up.resolution_size)) or size[0] != (r, r) or size[4] != (r, r) or size[3] != size[1] or any(a != b for a, b in size):
            return None
        scale, shift, scale_map, shift_map = self._normalizer_terms(r, X.device)
        keep = []

        ptr = lambda t: ops.kept_pointer(keep, t)
        m = DarcyModel()
        m.r, m.mid, m.ra, m.n_encoder, m.n_decoder = r, size[1][0], size[2][0], len(enc), len(dec.layers)
        m.d_pos = enc[0].attention_layer.dim_position if enc else dec.dim_position
        m.modes = dec.layers[0].mode if len(dec.layers) else 1
        m.c1, m.c2, m.c3 = down.dims
        m.act_down, m.act_dec = ops.act_code(down.activation), ops.act_code(dec.activation)
        m.act_up = ops.act_code('silu2' if up.activation == 'silu' else 'relu')
        m.act_ffn = ops.act_code(enc[0].ffn_layer.activation) if enc else 0
        m.eps = enc[0].attention_layer.norm_eps if enc else 0.0
        m.dirichlet = int(self.boundary_condition == 'dirichlet')
        m.scale, m.shift, m.scale_map, m.shift_map = scale, shift, ptr(scale_map), ptr(shift_map)
        m.conv0_w, m.conv0_b = ptr(down.kernel_weight0()), ptr(down.conv0.conv_layer.bias.detach())
        cin = 128
        for i, (conv, c) in enumerate(zip((down.conv1, down.conv2, down.conv3), down.dims)):
            w, b = conv.tc_weight(cin, (c + 3) // 4 * 4)
            m.conv_w[i], m.conv_b[i], cin = ptr(w), ptr(b), (c + 3) // 4 * 4
        for i, layer in enumerate(enc):
            layer.fill_native(m.encoder[i], ptr)
        w, b = up.conv.tc_weight(128, 128)
        m.up_w, m.up_b = ptr(w), ptr(b)
        wx, wg = dec._split_fc()
        m.fcx_w, m.fcg_w, m.fc_b = ptr(wx), ptr(wg), ptr(dec.spatial_fc_layer.bias.detach())
        for i, layer in enumerate(dec.layers):
            layer.fill_native(m.decoder[i], ptr)
        m.tables = ptr(ops.spectral_tables(r, m.modes, X.device).view(torch.float32)) if len(dec.layers) else None
        w1, w2 = dec.head_weights()
        m.head_w1, m.head_b1, m.head_w2 = ptr(w1), ptr(dec.ffn_layer.layer1.bias.detach()), ptr(w2)
        return ops.DarcyPlan(m, keep, ptr(dec.ffn_layer.layer2.bias.detach()))

    def _native_widths(self) -> bool:
        """Whether the one-call forward covers this model: its own module types, the widths the kernels are made for, and one
        activation and epsilon throughout."""
        enc, dec, down, up = self.encoder_mixer.layers, self.decoder_regressor, self.down_scaler, self.up_scaler
        if not (type(dec) is Sp_DecoderRegressor
                and all(type(l) is Sp_EncoderLayer for l in enc) and all(type(l) is Sp_SpectralConv2D for l in dec.layers)
                and all(type(c) is ConvResBlock2D for c in (down.conv0, down.conv1, down.conv2, down.conv3, up.conv))
                and type(up.conv.conv_layer) is torch.nn.Conv2d and type(dec.spatial_fc_layer) is torch.nn.Linear):
            return False
        return (all(l.fusable and l.attention_layer.norm_eps == enc[0].attention_layer.norm_eps
                    and l.ffn_layer.activation == enc[0].ffn_layer.activation for l in enc)
                and all(c.activation == down.activation for c in (down.conv1, down.conv2, down.conv3))
                and up.conv.conv_layer.in_channels == 128 and up.conv.conv_layer.out_channels == 128 and dec.in_dim == 128
                and dec.dim_position == 2 and dec.spatial_fc_layer.out_features == 32 and dec.ffn_layer.layer1.out_features == 128
                and all(l.structure == 'fused' and l.in_dim == 32 and l.out_dim == 32 and l.activation == dec.activation
                        and l.mode == dec.layers[0].mode for l in dec.layers))

    def _forward_modules(self, X: Tensor, position: Tensor, grid: Tensor, taps: dict = None) -> Tensor:
        r = X.shape[1]
        scale, shift, scale_map, shift_map = self._normalizer_terms(r, X.device)
        X = self.down_scaler(X)
        if taps is not None:
            taps['down'] = X
        N, ra, _, D = X.shape
        pos = position.reshape(N, ra * ra, position.size(-1))
        X = X.view(N, ra * ra, D)
        for i, layer in enumerate(self.encoder_mixer.layers):
            X = layer(X, pos)
            if taps is not None:
                taps[f'enc{i}'] = X
        U = self.up_scaler.forward_mid(X.view(N, ra, ra, D))
        if taps is not None:
            taps['up_mid'] = U
        return self.decoder_regressor.forward_from_mid(U, grid, scale, shift, self.boundary_condition == 'dirichlet',
                                                       scale_map, shift_map)
