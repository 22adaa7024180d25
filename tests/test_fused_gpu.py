"""The fused encoder-layer kernels and the shared-memory convolution kernel against float64, at the edges of their tiles."""
import pytest
import torch

from tests.helpers import rel_l2
from oracle import gt_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5          # per layer, as for the single ops


def _layer(seed):
    from spgt_b200.network.sp_layer import Sp_EncoderLayer
    g = torch.Generator().manual_seed(seed)
    layer = Sp_EncoderLayer(128, 4, 2, 1e-6, 0.0, 0.0, 1e-2, 1e-2, False, 256, 0.0, 'relu').eval()
    with torch.no_grad():
        for name, p in layer.named_parameters():
            scale = {1: 0.1, 2: p.shape[-1] ** -0.5}[p.dim()] if 'ln_' not in name else 0.1
            p.copy_(torch.randn(p.shape, generator=g) * scale + (1.0 if 'ln_weight' in name else 0.0))
    return layer, g


# one node, ends of a 128-row tile, one tile more than a sample needs, blocks that work on two samples, more tiles than blocks
@pytest.mark.parametrize('B,S', [(1, 1), (1, 127), (2, 128), (3, 129), (2, 641), (5, 1849), (80, 130), (64, 2809)])
def test_encoder_layer_edges(B, S):
    from spgt_b200 import ops
    layer, g = _layer(S)
    x, pos = torch.randn(B, S, 128, generator=g), torch.rand(B, S, 2, generator=g)
    n = min(B, 3)                                          # (the oracle runs on the first and last samples)
    idx = sorted({0, B // 2, B - 1})[:n]
    p = {k: v.detach().double().clone() for k, v in layer.state_dict().items()}
    cfg = dict(num_head=4, dim_hidden=128, attn_norm_eps=1e-6, acti_encoder_ffn='relu')
    taps = {}
    ref = O.encoder_layer(x[idx].double(), pos[idx].double(), p, '', cfg, taps)
    layer = layer.cuda()
    xd, pd = x.cuda(), pos.cuda()
    with torch.no_grad():
        y = layer(xd, pd)
        att = layer.attention_layer(xd, xd, xd, pd)
        res = layer.attention_layer(xd, xd, xd, pd, residual=xd)
        again = layer(xd, pd)
    assert ops.tc_status() == 0
    assert torch.equal(y, again) and torch.isfinite(y).all()
    assert rel_l2(y[idx], ref) < TOL
    assert rel_l2(att[idx], taps['fc']) < TOL
    assert rel_l2(res[idx], taps['post_attn']) < TOL


@pytest.mark.parametrize('B,Hh,Ww,Cin,Cout,act', [(1, 1, 1, 4, 4, None), (2, 9, 11, 128, 44, 'relu'), (1, 16, 8, 44, 44, 'silu'), (3, 17, 9, 36, 48, 'relu'),
                                                   (2, 15, 31, 12, 20, None), (3, 17, 9, 36, 64, 'relu'), (20, 77, 77, 44, 56, 'relu'), (1, 20, 17, 128, 128, 'silu2'), (2, 5, 106, 64, 52, 'silu'),
                                                   (4, 106, 106, 128, 128, 'silu2'), (20, 77, 77, 128, 44, 'relu')])
def test_conv3x3_shared_memory_operands(B, Hh, Ww, Cin, Cout, act):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(Hh * Ww + Cout)
    x, w, b = torch.randn(B, Hh, Ww, Cin + 8, generator=g), torch.randn(Cout, Cin, 3, 3, generator=g) / (9 * Cin) ** 0.5, torch.randn(Cout, generator=g)
    wt = ops.ConvWeight(w.permute(2, 3, 1, 0).reshape(9 * Cin, Cout).contiguous().cuda(), Cin)
    y = torch.full((B, Hh, Ww, Cout + 8), float('nan'), device='cuda')
    ops.conv3x3_tc(x.cuda(), 4, Cin, wt, b.cuda(), y, 4, Cout, act)
    assert ops.tc_status() == 0
    ref = torch.nn.functional.conv2d(x[..., 4:4 + Cin].permute(0, 3, 1, 2).double(), w.double(), b.double(), padding=1)
    silu = torch.nn.functional.silu
    ref = {None: lambda t: t, 'relu': torch.relu, 'silu': silu, 'silu2': lambda t: silu(silu(t))}[act](ref)
    assert rel_l2(y[..., 4:4 + Cout], ref.permute(0, 2, 3, 1)) < TOL
    assert torch.isnan(y[..., :4]).all() and torch.isnan(y[..., 4 + Cout:]).all()


# rows: one, around a 32-row block, around the 256 rows from which two blocks share them, many blocks; widths: tails of the 128-wide tiles
@pytest.mark.parametrize('rows,M,N', [(1, 4, 4), (31, 128, 128), (33, 132, 36), (257, 128, 256), (1000, 256, 128), (7396, 136, 128), (65536, 128, 128), (79524, 32, 128)])
def test_weight_gradient_gemm(rows, M, N):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(rows)
    a, b = torch.randn(rows, M, generator=g), torch.randn(rows, N, generator=g)
    c, s = ops.tn_gemm(a.cuda(), b.cuda(), column_sums=True)
    assert ops.tc_status() == 0
    # sums of `rows` products of independent entries: fp32 accumulation errors grow with the square root of their number, as the sums do
    assert rel_l2(c, a.double().t() @ b.double()) < TOL
    assert rel_l2(s, b.double().sum(0)) < TOL
    c2, s2 = ops.tn_gemm(a.cuda(), b.cuda(), column_sums=True)
    assert torch.equal(c, c2) and torch.equal(s, s2)


@pytest.mark.parametrize('norm', [False, True])
def test_projection_backward_takes_any_alignment(norm):
    """x, and h and dh of the element-wise entry point, may start at any float."""
    from spgt_b200 import ops
    from spgt_b200._lib import lib
    g = torch.Generator().manual_seed(9)
    shifted = lambda t: torch.empty(t.numel() + 1, device='cuda')[1:].view(t.shape).copy_(t)
    B, S = 2, 70
    x, w, b, dy = torch.randn(B, S, 128, generator=g).cuda(), torch.randn(128, 128, generator=g).cuda(), torch.randn(128, generator=g).cuda(), torch.randn(B, 4, 34, S, generator=g).cuda()
    if not norm:
        want = ops.projpos_backward(x, w, b, None, dy, 0.0, 4, 32, 2)
        got = ops.projpos_backward(shifted(x), w, b, None, dy, 0.0, 4, 32, 2)
        assert all(torch.equal(p, q) for p, q in zip(want[:3], got[:3]))
    h, lnw = torch.randn(B * S, 128, generator=g).cuda(), torch.randn(4, 32, generator=g).cuda() if norm else None
    need = int(lib.spgt_projpos_bwd_workspace_bytes(B, S, 4))
    runs = []
    for place in (torch.clone, shifted):
        hh, dh, sums, ws = place(h), place(torch.zeros_like(h)), torch.zeros(3, 128, device='cuda'), torch.empty(need, dtype=torch.uint8, device='cuda')
        code = lib.spgt_projpos_bwd_elementwise(dy.data_ptr(), hh.data_ptr() if norm else None, lnw.data_ptr() if norm else None, 1e-6, dh.data_ptr(), *(s.data_ptr() for s in sums),
                                                B, S, 4, 32, 2, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
        assert code == 0
        runs.append((dh, sums))
    assert all(torch.equal(p, q) for p, q in zip(*runs))


# the kernel stands in for fp32 products from 128 rows on: no further from fp64 than they are (a tenth more for the scatter of one draw),
# for entries of both signs and for entries of one, where truncated sums would drift
@pytest.mark.parametrize('one_sign', [False, True])
@pytest.mark.parametrize('rows,M,N', [(128, 128, 256), (200, 256, 128), (1849, 128, 136), (7396, 128, 256), (65536, 256, 128)])
def test_weight_gradient_gemm_is_as_close_as_fp32(rows, M, N, one_sign):
    from spgt_b200 import ops
    torch.backends.cuda.matmul.allow_tf32 = False
    g = torch.Generator().manual_seed(rows)
    draw = torch.rand if one_sign else torch.randn
    a, b = draw(rows, M, generator=g).cuda(), draw(rows, N, generator=g).cuda()
    want = a.double().t() @ b.double()
    assert rel_l2(ops.tn_gemm(a, b)[0], want) <= 1.1 * rel_l2(a.t() @ b, want)


def _model():
    from spgt_b200.config.config_accessor import get_darcy_config
    from spgt_b200.dataset.darcy_dataset import GaussNormalizer, meshgrid
    from spgt_b200.network.sp_model import Sp_GalerkinTransformer2D
    cfg = get_darcy_config(3, 6, num_frequence_mode=4, clamp_attn=False, fine_resolution=85, num_encoder_layer=2)
    cfg['target_normalizer'] = GaussNormalizer()
    torch.manual_seed(5)
    model = Sp_GalerkinTransformer2D(cfg).cuda().eval()
    g = torch.Generator().manual_seed(6)
    expand = lambda m: torch.from_numpy(m).float().expand(3, *m.shape).contiguous().cuda()
    return model, torch.randn(3, 29, 29, 1, generator=g).cuda(), expand(meshgrid(85, 6)), expand(meshgrid(85, 3))


def test_one_call_forward_yields_to_observed_or_changed_modules():
    import copy
    model, *args = _model()
    ref = model(*args)
    assert torch.equal(copy.deepcopy(model)(*args), ref)           # a copy makes its own plan
    seen = []
    handles = [m.register_forward_hook(lambda m, i, o: seen.append(type(m).__name__))
               for m in (model.encoder_mixer.layers[1].ffn_layer, model.decoder_regressor.layers[0], model.encoder_mixer.layers[0])]
    assert rel_l2(model(*args), ref) < TOL
    assert sorted(seen) == ['FeedForward', 'Sp_EncoderLayer', 'Sp_SpectralConv2D']
    for h in handles:
        h.remove()
    assert torch.equal(model(*args), ref)

    class Twice(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, x, position):
            return self.inner(self.inner(x, position), position)
    class Scaler(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, x):
            return self.inner(x)

        def forward_mid(self, x):
            return self.inner.forward_mid(x)
    for name in ('down_scaler', 'up_scaler'):
        inner = getattr(model, name)
        setattr(model, name, Scaler(inner))
        assert rel_l2(model(*args), ref) < TOL
        setattr(model, name, inner)
    plain = model.encoder_mixer.layers[1]
    model.encoder_mixer.layers[1] = Twice(plain)
    twice = model(*args)
    model.encoder_mixer.layers[1] = plain
    model.encoder_mixer.layers.append(plain)
    assert rel_l2(twice, model(*args)) < TOL
    model.encoder_mixer.layers = model.encoder_mixer.layers[:2]
    for layer in model.encoder_mixer.layers:
        layer.attention_layer.norm_eps = 0.5                       # an option set after the first forward counts
    assert rel_l2(model(*args), ref) > 1e-3


def test_encoder_layer_training_differentiates_twice():
    """A penalty on one weight's gradient: its own gradients go through the layer's backward and forward pass."""
    layer, g = _layer(11)
    x, pos = torch.randn(2, 45, 128, generator=g), torch.rand(2, 45, 2, generator=g)
    p = {k: v.detach().double().requires_grad_() for k, v in layer.state_dict().items()}
    cfg = dict(num_head=4, dim_hidden=128, attn_norm_eps=1e-6, acti_encoder_ffn='relu')
    xr = x.double().requires_grad_()

    def penalty(y, weight):
        grad, = torch.autograd.grad(y.square().mean(), weight, create_graph=True)
        return grad.square().sum()
    w2 = 'ffn_layer.layer2.weight'
    names = ['attention_layer.weight_K', 'attention_layer.fc_layer.weight', w2]
    want = torch.autograd.grad(penalty(O.encoder_layer(xr, pos.double(), p, '', cfg), p[w2]), [xr, *(p[n] for n in names)])
    layer = layer.cuda().train()
    dev, xd = dict(layer.named_parameters()), x.cuda().requires_grad_()
    got = torch.autograd.grad(penalty(layer.forward_train(xd, pos.cuda()), dev[w2]), [xd, *(dev[n] for n in names)])
    for n, a, b in zip(['x'] + names, got, want):
        assert rel_l2(a, b) < TOL, n


def test_encoder_layer_training_without_a_projection_bias():
    layer, g = _layer(13)
    x, pos = torch.randn(2, 45, 128, generator=g), torch.rand(2, 45, 2, generator=g)
    with torch.no_grad():
        layer.attention_layer.bias_K.zero_()
    layer = layer.cuda().train()
    with torch.no_grad():
        ref = layer.forward_train(x.cuda(), pos.cuda())
        layer.attention_layer.bias_K = None
        assert rel_l2(layer.forward_train(x.cuda(), pos.cuda()), ref) < TOL


def test_single_entry_points_can_be_timed():
    from spgt_b200 import ops
    model, *args = _model()
    ref = model(*args)
    with ops.profile_ops() as profile:
        out = model(*args)
    times = profile.times_ms()
    assert len(times['spgt_encoder_layer_fwd']) == 2 and len(times['spgt_spectral_conv2d_fwd']) == 2 and 'spgt_darcy_forward_devbias' not in times
    assert rel_l2(out, ref) < TOL and torch.equal(model(*args), ref)


def test_one_call_forward_yields_to_other_grids():
    """A grid of other nodes (the regressor is evaluated there), or one with more samples than there are fields."""
    from spgt_b200.dataset.darcy_dataset import meshgrid
    model, node, position, grid = _model()
    ref = model(node, position, grid)
    assert torch.equal(model(node[:2], position[:2], grid), ref[:2])
    other = torch.from_numpy(meshgrid(57, 1)).float().expand(3, 57, 57, 2).contiguous()
    out = model(node, position, other.cuda())
    cfg = O.default_config(85, 3, 6, 4, 2, 2)
    cfg['resolution_size'] = [*cfg['resolution_size'][:4], (57, 57)]
    want = O.model_forward(node.cpu().double(), position.cpu().double(), other.double(), O.to_dtype(model.cpu().state_dict(), torch.float64), cfg)
    assert rel_l2(out, want) < TOL
    with pytest.raises((ValueError, RuntimeError)):
        model.cuda()(node.squeeze(-1), position, grid)          # (the fields have a channel dimension)


@pytest.mark.parametrize('training', [False, True])
def test_encoder_layer_takes_positions_of_any_leading_shape(training):
    layer, g = _layer(5)
    layer = layer.cuda().train(training)
    x, pos = torch.randn(2, 49, 128, generator=g).cuda(), torch.rand(3, 49, 2, generator=g).cuda()
    run = layer.forward_train if training else layer
    with torch.no_grad():
        ref = run(x, pos[:2].contiguous())
        assert torch.equal(run(x, pos[:2].view(2, 7, 7, 2)), ref) and torch.equal(run(x, pos), ref)
        with pytest.raises(ValueError):
            run(x, pos[:1].contiguous())


def test_encoder_layer_takes_any_dense_or_strided_weights_and_positions():
    layer, g = _layer(3)
    x, pos = torch.randn(2, 45, 128, generator=g).cuda(), torch.rand(2, 45, 2, generator=g).cuda()
    layer = layer.cuda()
    with torch.no_grad():
        ref = layer(x, pos)
        shifted = torch.empty(2 * 45 * 2 + 1, device='cuda')[1:].view(2, 45, 2).copy_(pos)
        assert torch.equal(layer(x, shifted), ref)
        assert torch.equal(layer(x[1:], pos[1:]), layer(x[1:].clone(), pos[1:].clone()))
        a = layer.attention_layer
        a.weight_Q.data = a.weight_Q.data.t().contiguous().t()
        a.weight_K.data = a.weight_K.data.t().contiguous().t()
        w = a.fc_layer.weight.data
        a.fc_layer.weight.data = torch.empty(w.numel() + 1, device='cuda')[1:].view_as(w).copy_(w)
        assert torch.equal(layer(x, pos), ref)


# slices of the x transforms: none, one with a remainder, as many as rows or modes allow; grids of one, two and three 256-row units
@pytest.mark.parametrize('B,r,m', [(1, 2, 1), (1, 95, 12), (1, 97, 12), (1, 256, 16), (2, 257, 16), (2, 421, 15), (3, 513, 3), (1, 600, 16), (20, 150, 8), (70, 40, 5)])
def test_spectral_layer_slices_and_units(B, r, m):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(r + m)
    x = torch.randn(B, r, r, 32, generator=g)
    p = {'residual_layer.weight': torch.randn(32, 32, generator=g) / 6, 'residual_layer.bias': torch.randn(32, generator=g),
         'fourier_weight.0': torch.randn(m, m, 32, 32, 2, generator=g) / 6, 'fourier_weight.1': torch.randn(m, m, 32, 32, 2, generator=g) / 6}
    dev = {k: v.cuda() for k, v in p.items()}
    args = (dev['residual_layer.weight'].t().contiguous(), dev['residual_layer.bias'], dev['fourier_weight.0'], dev['fourier_weight.1'], m, 'silu')
    y = ops.spectral_conv2d(x.cuda(), *args)
    assert ops.tc_status() == 0
    idx = sorted({0, B - 1})
    ref = O.spectral_conv2d(x[idx].double(), O.to_dtype(p, torch.float64), '', m, 'silu')
    assert rel_l2(y[idx], ref) < TOL
    assert torch.equal(y, ops.spectral_conv2d(x.cuda(), *args))


# columns around the 112-wide tiles, 16-byte and 4-byte copies, several chunks and blocks of several tiles
@pytest.mark.parametrize('B,H,dpk,S', [(1, 1, 34, 1), (2, 4, 34, 111), (1, 4, 34, 112), (3, 2, 35, 113), (16, 4, 34, 4096), (2, 3, 32, 4097), (80, 4, 34, 225), (300, 4, 34, 16), (3, 2, 1, 500), (2, 3, 12, 300), (2, 3, 13, 1000), (1, 2, 24, 63), (1, 2, 25, 130)])
def test_attention_backward_tiles(B, H, dpk, S):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, dpk, S, generator=g).cuda() for _ in range(3))
    dout = torch.randn(B, H, S, dpk, generator=g).cuda()
    Q, K, V = (t.double().requires_grad_() for t in (q, k, v))
    want = torch.autograd.grad(Q.transpose(2, 3) @ (K @ V.transpose(2, 3) / S), [Q, K, V], dout.double())
    got = ops.galerkin_attention_backward(q, k, v, dout)
    for n, a, b in zip('QKV', got, want):
        assert rel_l2(a, b) < TOL, n
    assert all(torch.equal(a, b) for a, b in zip(got, ops.galerkin_attention_backward(q, k, v, dout)))


# one node, both sides of the 128 rows from which the weight-gradient kernel runs, samples that share its 32-row blocks
@pytest.mark.parametrize('B,S', [(1, 1), (1, 127), (1, 128), (2, 129), (3, 171), (4, 1849), (40, 33)])
def test_encoder_layer_training_gradients(B, S):
    from spgt_b200 import ops
    layer, g = _layer(S)
    x, pos, dy = torch.randn(B, S, 128, generator=g), torch.rand(B, S, 2, generator=g), torch.randn(B, S, 128, generator=g)
    p = {k: v.detach().double().requires_grad_() for k, v in layer.state_dict().items()}
    xr = x.double().requires_grad_()
    cfg = dict(num_head=4, dim_hidden=128, attn_norm_eps=1e-6, acti_encoder_ffn='relu')
    names = [n for n, _ in layer.named_parameters()]
    layer = layer.cuda().train()
    xd = x.cuda().requires_grad_()
    taps = {}
    O.encoder_layer(xr, pos.double(), p, '', cfg, taps)
    x1, linear = taps['post_attn'], torch.nn.functional.linear
    runs = []
    for _ in range(2):
        y = layer.forward_train(xd, pos.cuda())
        runs.append((y, *torch.autograd.grad(y, [xd] + list(layer.parameters()), dy.cuda())))
    y = layer.forward_train(xd, pos.cuda())
    passes = y.grad_fn.saved_tensors[2].cpu() > 0
    w1 = p['ffn_layer.layer1.weight']
    pre = linear(x1, w1, p['ffn_layer.layer1.bias'])
    # a value within rounding of zero may pass the ReLU there and not in float64: x1 is within TOL of its row's norm
    rounding = TOL * x1.norm(dim=-1, keepdim=True) * w1.norm(dim=1)
    assert bool(((passes == (pre > 0)) | (pre.abs() < rounding)).all())
    h = pre * passes
    ref = x1 + linear(h, p['ffn_layer.layer2.weight'], p['ffn_layer.layer2.bias'])
    want = torch.autograd.grad(ref, [xr] + [p[n] for n in names], dy.double())
    assert ops.tc_status() == 0 and y.grad_fn.name().startswith('_EncoderLayerFunction')
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    assert rel_l2(runs[0][0], ref.detach()) < TOL
    for n, a, b in zip(['x'] + names, runs[0][1:], want):
        assert rel_l2(a, b) < 2 * TOL, n
    handle = layer.ffn_layer.layer1.register_forward_hook(lambda m, i, o: None)      # an observed layer runs op by op
    y = layer.forward_train(xd, pos.cuda())
    handle.remove()
    assert not y.grad_fn.name().startswith('_EncoderLayerFunction') and rel_l2(y, runs[0][0]) < TOL


def test_encoder_layer_training_runs_backward_hooks():
    """Hooks on the linear layers see, and may change, the gradients as they do op by op."""
    layer, g = _layer(7)
    layer = layer.cuda().train()
    x, pos, dy = torch.randn(2, 45, 128, generator=g).cuda().requires_grad_(), torch.rand(2, 45, 2, generator=g).cuda(), torch.randn(2, 45, 128, generator=g).cuda()
    plain = torch.autograd.grad(layer.forward_train(x, pos), layer.attention_layer.fc_layer.bias, dy)[0]
    seen = []
    members = (layer.attention_layer.fc_layer, layer.ffn_layer.layer1, layer.ffn_layer.layer2)
    handles = [m.register_full_backward_hook(lambda m, gi, go: seen.append(m)) for m in members]
    handles.append(members[0].register_full_backward_pre_hook(lambda m, go: (2 * go[0],)))
    hooked = torch.autograd.grad(layer.forward_train(x, pos), [x, members[0].bias], dy)[1]
    assert {id(m) for m in seen} == {id(m) for m in members}
    assert rel_l2(hooked, 2 * plain) < TOL
    for h in handles:
        h.remove()
    assert torch.equal(torch.autograd.grad(layer.forward_train(x, pos), members[0].bias, dy)[0], plain)


# ragged segments, one pixel, channel counts that fill a block, divide it unevenly or exceed it
@pytest.mark.parametrize('B,Hi,Ho,c', [(1, 5, 1, (2, 1, 1)), (2, 77, 43, (42, 42, 44)), (64, 19, 9, (42, 42, 44)), (1, 31, 50, (100, 101, 99)), (3, 8, 8, (5, 6, 9))])
def test_bilinear_concat3(B, Hi, Ho, c):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(Hi)
    pad = lambda n: (n + 3) // 4 * 4
    x = [torch.randn(B, Hi, Hi, pad(n), generator=g) for n in c]
    y = ops.bilinear_concat3(*[t.cuda() for t in x], *c, Ho, Ho, 'relu')
    cat = torch.cat([t[..., :n] for t, n in zip(x, c)], dim=-1).permute(0, 3, 1, 2)
    ref = torch.relu(torch.nn.functional.interpolate(cat, size=(Ho, Ho), mode='bilinear', align_corners=True)).permute(0, 2, 3, 1)
    assert rel_l2(y, ref) < 1e-6          # (the same fp32 source coordinates, four products and three sums)


def test_images_from_the_modules_weights():
    """Prepared in one launch from the weights as they are: the same bits as from rearranged copies (K / V: but for the rounding of the mean)."""
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(8)
    wk, wv, w1, w2 = (torch.randn(*s, generator=g).cuda() for s in ((128, 128), (128, 128), (256, 128), (128, 256)))
    images, alone = ops.EncoderImages(wk, wv, w1, w2), ops.EncoderImages(wk, wv)
    parts = images.buf.view(3, -1)
    assert torch.equal(parts[0], alone.buf)
    for part, w in zip(parts[1:], (w1, w2)):
        assert torch.equal(part, ops.TcWeight(w, transposed=True).buf)
    w = torch.stack([wk, wv], dim=1).double().view(128, 2, 4, 32)
    w = (w - w.mean(dim=3, keepdim=True)).view(128, 2, 2, 64).transpose(1, 2).reshape(128, 256)
    got, want = (t.view(torch.float32).view(2, 4, 2, -1).double().sum(2) for t in (parts[0], ops.TcWeight(w.float()).buf))      # hi + lo
    assert rel_l2(got, want) < 2e-7                      # one ulp of the mean of 32 values
    for cin, cout, cin_pad, cout_pad in ((128, 42, 128, 44), (42, 42, 44, 44), (1, 3, 4, 4), (66, 50, 68, 64), (128, 128, 128, 128)):
        w, b = torch.randn(cout, cin, 3, 3, generator=g).cuda(), torch.randn(cout, generator=g).cuda()
        pad = torch.zeros(cout_pad, cin_pad, 3, 3, device='cuda')
        pad[:cout, :cin] = w
        prepared, bias = ops.ConvWeight.padded(w, b, cin_pad, cout_pad)
        assert torch.equal(prepared.buf, ops.ConvWeight(pad.permute(2, 3, 1, 0).reshape(9 * cin_pad, cout_pad).contiguous(), cin_pad).buf)
        assert torch.equal(bias, torch.nn.functional.pad(b, (0, cout_pad - cout)))


def _with_nan(t, at):
    """t with a NaN as arithmetic on the GPU makes it (all mantissa bits set)."""
    t = t.clone()
    t.view(torch.int32).view(-1)[at] = 0x7fffffff
    return t


# one not-a-number in one operand: the values that depend on it, and no others, are NaN
@pytest.mark.parametrize('which', ['x', 'weight', 'bias'])
def test_projection_passes_nan_on(which):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(2)
    t = {'x': torch.randn(1, 150, 128, generator=g), 'weight': torch.randn(128, 128, generator=g), 'bias': torch.randn(128, generator=g)}
    t[which] = _with_nan(t[which], 77)
    out = ops.projpos(*(v.cuda() for v in t.values()), torch.zeros(1, 150, 2).cuda(), 4, 32, 2)[0, :, 2:]
    want = (t['x'][0] @ t['weight'] + t['bias']).t().reshape(4, 32, 150)
    assert torch.equal(torch.isnan(out.cpu()), torch.isnan(want))


@pytest.mark.parametrize('which', [0, 1, 2])
def test_attention_passes_nan_on(which):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(3)
    t = [torch.randn(1, 4, 34, 150, generator=g) for _ in range(3)]
    t[which] = _with_nan(t[which], 5000)
    q, k, v = t
    out = ops.galerkin_attention(*(a.cuda() for a in t))
    assert torch.equal(torch.isnan(out.cpu()), torch.isnan(q.transpose(2, 3) @ (k @ v.transpose(2, 3))))


@pytest.mark.parametrize('r', [40, 260])
@pytest.mark.parametrize('which', ['x', 'mode', 'residual'])
def test_spectral_layer_passes_nan_on(r, which):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(4)
    x, w = torch.randn(2, r, r, 32, generator=g), torch.randn(32, 32, generator=g)
    fw = [torch.randn(4, 4, 32, 32, 2, generator=g) for _ in range(2)]
    nan = torch.zeros(2, r, r, 32, dtype=torch.bool)
    if which == 'x':
        x, nan[1] = _with_nan(x, r * r * 32 + 100), True
    elif which == 'mode':
        fw[1], nan[..., 5] = _with_nan(fw[1], 2 * (32 * 40 + 5)), True
    else:
        w, nan[..., 7] = _with_nan(w, 32 * 3 + 7), True
    out = ops.spectral_conv2d(x.cuda(), w.cuda(), torch.zeros(32).cuda(), fw[0].cuda(), fw[1].cuda(), 4, None)
    assert torch.equal(torch.isnan(out.cpu()), nan)


@pytest.mark.parametrize('which', [0, 1])
def test_weight_gradient_gemm_passes_nan_on(which):
    from spgt_b200 import ops
    g = torch.Generator().manual_seed(6)
    t = [torch.randn(3000, 128, generator=g), torch.randn(3000, 36, generator=g)]
    t[which] = _with_nan(t[which], 5000)
    c, sums = ops.tn_gemm(*(a.cuda() for a in t), column_sums=True)
    assert torch.equal(torch.isnan(c.cpu()), torch.isnan(t[0].t() @ t[1])) and torch.equal(torch.isnan(sums.cpu()), torch.isnan(t[1].sum(0)))


# both sides of the rule: many samples of few nodes run on the single ops, the same samples a few at a time on the fused kernels
@pytest.mark.parametrize('B,S,single', [(300, 40, True), (250, 129, True), (100, 129, False), (260, 250, False)])
def test_encoder_layer_route(B, S, single):
    from spgt_b200 import ops
    layer, g = _layer(S)
    layer = layer.cuda()
    x, pos = torch.randn(B, S, 128, generator=g).cuda(), torch.rand(B, S, 2, generator=g).cuda()
    with torch.no_grad():
        with ops.profile_ops() as profile:
            y = layer(x, pos)
        assert ('spgt_encoder_layer_fwd' not in profile.times_ms()) == single
        assert rel_l2(y[:20], layer(x[:20], pos[:20])) < TOL and rel_l2(y[-20:], layer(x[-20:], pos[-20:])) < TOL
        with pytest.raises(ValueError):
            layer(x, pos[:-1])
    assert ops.tc_status() == 0


@pytest.mark.parametrize('B,R,general', [(400, 9, True), (2000, 3, True), (8, 9, False), (64, 17, False)])
def test_convolution_route(B, R, general):
    from spgt_b200 import ops
    from spgt_b200.network.layer import ConvResBlock2D
    torch.manual_seed(R)
    block = ConvResBlock2D(20, 44, 3, 1, 0.0, 'relu').cuda()
    x = torch.randn(B, R, R, 20, device='cuda')
    with torch.no_grad(), ops.profile_ops() as profile:
        y = block.forward_tc(x, 20, 44)
    assert ('spgt_conv3x3_tc_fwd' in profile.times_ms()) == general
    ref = torch.nn.functional.conv2d(x.cpu().permute(0, 3, 1, 2).double(), block.conv_layer.weight.cpu().double(), block.conv_layer.bias.cpu().double(), padding=1)
    assert rel_l2(y, torch.relu(ref).permute(0, 2, 3, 1).detach()) < TOL


def test_model_of_many_small_fields_runs_module_by_module():
    from spgt_b200 import ops
    model, node, position, grid = _model()                       # 15 x 15 attention nodes
    times = lambda t: t[torch.arange(200) % 3].contiguous()
    ref = model(node, position, grid)
    before = ops.LAUNCHES
    out = model(times(node), times(position), times(grid))
    assert rel_l2(out, ref[torch.arange(200) % 3]) < TOL and ops.LAUNCHES > before
    assert not model._native_shapes(times(node), times(position), times(grid)) and model._native_shapes(node, position, grid)
