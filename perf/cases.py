"""What the performance of this framework is measured on: the Darcy Galerkin Transformer in inference and training, and
the layers and ops that a host program calls on their own, from one field at a time to the full batch.

A case is a dict of plain values; `prepare` makes what a user's program has in hand before the call, `run` is one pass
through the public entry points.
"""
import math

import torch

from spgt_b200.config.config_accessor import get_darcy_config
from spgt_b200.dataset.darcy_dataset import GaussNormalizer, meshgrid
from spgt_b200.engine.darcy_engine import HostInference
from spgt_b200.engine.metric import WeightedL2Loss2D
from spgt_b200.engine.train import train_epoch_darcy
from spgt_b200.extension.bind.galerkin_attention import (batched_skinny_gemm, multihead_galerkin_attention_cccr_cuda,
                                                         multihead_projection_layernorm_with_position_rrc_cuda,
                                                         multihead_projection_with_position_rrc_cuda)
from spgt_b200.network.sp_layer import Sp_GalerkinAttention, Sp_SpectralConv2D
from spgt_b200.network.sp_model import Sp_GalerkinTransformer2D

HEADS, HEAD_DIM, HIDDEN, POS = 4, 32, 128, 2


def _model_case(kind, batch, fine, sub_node, sub_attn, modes, **more):
    return dict(kind=kind, batch=batch, fine=fine, sub_node=sub_node, sub_attn=sub_attn, modes=modes, **more)


def listed():
    return [
        # one coefficient field at a time, the interactive use of a trained operator: 141 x 141 nodes, 43 x 43 attention grid
        dict(_model_case('infer', 1, 421, 3, 10, 12), name='infer_b1_r141'),
        # the reference's own validation batch at its default sub-sampling
        dict(_model_case('infer', 4, 421, 3, 10, 12), name='infer_b4_r141'),
        # one GPU's share of a batch of 64 spread over eight GPUs, 211 x 211 nodes, 53 x 53 attention grid
        dict(_model_case('infer', 8, 421, 2, 8, 12), name='infer_b8_r211'),
        # the throughput benchmark: the whole batch of 64 on one GPU
        dict(_model_case('infer', 64, 421, 2, 8, 12), name='infer_b64_r211'),
        # super-resolution evaluation: every node of the 421 grid, 106 x 106 attention grid, 15 modes
        dict(_model_case('infer', 2, 421, 1, 4, 15), name='infer_b2_r421'),
        # serving from host memory: pinned batches in, pinned predictions out, forward replayed as a graph
        dict(_model_case('host', 16, 421, 2, 8, 12, batches=4), name='host_4xb16_r211'),
        # one optimisation step at the reference's training batch: forward, loss, backward, clipping, Adam
        dict(_model_case('train', 4, 421, 3, 10, 12), name='train_b4_r141'),
        # the attention layer alone, dropped into another program's network: 43 x 43 nodes, batch 4
        dict(kind='attn_layer', batch=4, nodes=1849, name='attn_layer_b4_n1849'),
        # the reference-named attention ops under autograd, forward and backward, 64 x 64 nodes
        dict(kind='attn_ops_grad', batch=16, nodes=4096, name='attn_ops_grad_b16_n4096'),
        # projection + LayerNorm + position op at a large node count (128 x 128), no gradients
        dict(kind='projpos', batch=16, nodes=16384, name='projpos_lnorm_b16_n16384'),
        # split-K products K^T V of 16 samples x 4 heads over 141 x 141 nodes
        dict(kind='skinny', batch=64, width=32, nodes=19881, name='skinny_b64_n19881'),
        # a Fourier layer alone: 211 x 211, width 32, 12 modes, batch 8
        dict(kind='spectral', batch=8, r=211, modes=12, name='spectral_b8_r211'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most):
    """Fine grid, sub-sampling and modes of a model: whole grids of any size, or the 421 grid sub-sampled."""
    if rng.random() < 0.5:
        sub = rng.choice([s for s in (1, 2, 3, 4, 5, 6, 7, 10) if 420 // s + 1 <= most])
        fine, r = 421, 420 // sub + 1
    else:
        sub, fine = 1, _log(rng, 32, min(most, 330))
        r = fine
    sub_attn = sub * rng.choice((2, 3, 4)) if r > 96 else sub * 2
    return fine, sub, sub_attn, r, min(16, math.ceil(math.sqrt(r)))


def draw(rng):
    kind = rng.choice(['infer'] * 6 + ['host', 'train', 'train', 'attn_layer', 'attn_ops_grad', 'projpos', 'skinny', 'spectral'])
    if kind in ('infer', 'host', 'train'):
        fine, sub, sub_attn, r, modes = _grid(rng, 141 if kind == 'train' else 421)
        cells = {'infer': 64 * 211 * 211, 'host': 16 * 211 * 211, 'train': 4 * 141 * 141}[kind]
        batch = _log(rng, 1, max(1, min(16 if kind == 'train' else 64, cells // (4 * r * r) if sub_attn < 4 * sub else cells // (r * r))))
        more = dict(batches=rng.choice((2, 3, 4))) if kind == 'host' else {}
        return _model_case(kind, batch, fine, sub, sub_attn, modes, **more)
    if kind == 'spectral':
        r = _log(rng, 29, 421)
        return dict(kind=kind, batch=_log(rng, 1, max(1, min(64, 16 * 211 * 211 // (r * r)))), r=r, modes=min(16, math.ceil(math.sqrt(r))))
    nodes = rng.choice([_log(rng, 200, 65536), _log(rng, 15, 256) ** 2])
    most = {'attn_layer': 16 * 4096, 'attn_ops_grad': 16 * 4096, 'projpos': 16 * 16384, 'skinny': 64 * 19881}[kind]
    batch = _log(rng, 1, max(1, min(64, most // nodes)))
    if kind == 'skinny':
        return dict(kind=kind, batch=batch, width=rng.choice((32, 34)), nodes=nodes)
    return dict(kind=kind, batch=batch, nodes=min(nodes, most))


# ------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator('cuda').manual_seed(seed)


def _fields(n, S, g, modes=48):
    """Coefficient fields: a Gaussian random field with covariance (-Laplace + 9)^-2 (cosine modes, the high ones, which
    carry nothing visible, left out), thresholded to 12 and 3.  [n, S, S]"""
    k = torch.arange(modes, device='cuda', dtype=torch.float32)
    x = (torch.arange(S, device='cuda', dtype=torch.float32) + 0.5) / S
    basis = torch.cos(math.pi * k[:, None] * x[None, :])
    coef = 1.0 / (math.pi ** 2 * (k[:, None] ** 2 + k[None, :] ** 2) + 9.0)
    coef[0, 0] = 0.0
    u = torch.einsum('nij,ix,jy->nxy', torch.randn(n, modes, modes, device='cuda', generator=g) * coef, basis, basis)
    return torch.where(u >= 0, 12.0, 3.0)


def _config(case):
    cfg = get_darcy_config(case['sub_node'], case['sub_attn'], num_frequence_mode=case['modes'], clamp_attn=False,
                           fine_resolution=case['fine'])
    cfg['target_normalizer'] = GaussNormalizer()
    return cfg


def _model(cfg, seed):
    torch.manual_seed(seed)
    with torch.device('cuda'):
        model = Sp_GalerkinTransformer2D(cfg)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if 'fourier_weight' in name:
                p.mul_(30.0)                 # trained Fourier weights contribute visibly, freshly drawn ones do not
    return model


def _batch(case, cfg, n, g):
    a = _fields(n, case['fine'], g)[:, ::case['sub_node'], ::case['sub_node']].unsqueeze(-1).contiguous()
    expand = lambda m: torch.from_numpy(m).float().cuda().expand(n, *m.shape).contiguous()
    return dict(coeff=a, node=(a - 7.5) / (4.5 + 1e-5), position=expand(meshgrid(case['fine'], cfg['subsample_attn'])),
                grid=expand(meshgrid(case['fine'], case['sub_node'])))


def _positions(batch, nodes, g):
    return torch.rand(batch, nodes, POS, device='cuda', generator=g)


def _projection(g):
    def normal(*shape, scale=1.0):
        return torch.randn(*shape, device='cuda', generator=g) * scale
    return [normal(HIDDEN, HIDDEN, scale=HIDDEN ** -0.5), normal(HIDDEN, scale=0.1), 1.0 + normal(HEADS, HEAD_DIM, scale=0.1),
            normal(HEADS, HEAD_DIM, scale=0.1)]


def prepare(case, seed):
    kind, g = case['kind'], _generator(seed)
    if kind in ('infer', 'host', 'train'):
        cfg = _config(case)
        model = _model(cfg, seed)
        n = case['batch']
        if kind == 'infer':
            return dict(kind=kind, model=model.eval(), **_batch(case, cfg, n, g))
        if kind == 'host':
            data = [_batch(case, cfg, n, g) for _ in range(case['batches'])]
            fixed = {k: data[0][k].cpu().pin_memory() for k in ('position', 'grid')}
            batches = [dict(node=d['node'].cpu().pin_memory(), **fixed) for d in data]
            engine = HostInference(model.eval(), 'cuda', use_graphs=True, static_keys=('position', 'grid'))
            return dict(kind=kind, engine=engine, batches=batches)
        # training computes in fp32 throughout, as the rest of the framework does
        torch.backends.cudnn.allow_tf32 = False
        torch.backends.cuda.matmul.allow_tf32 = False
        batch = _batch(case, cfg, n, g)
        r = cfg['r_node']
        smooth = torch.sin(math.pi * batch['grid'][..., :1]) * torch.sin(math.pi * batch['grid'][..., 1:])
        batch['target'] = 0.02 * smooth * (1.0 + 0.2 * torch.rand(n, 1, 1, 1, device='cuda', generator=g))
        batch['target_grad'] = 0.06 * torch.randn(n, r, r, 2, device='cuda', generator=g)
        return dict(kind=kind, model=model, batch=batch, loss=WeightedL2Loss2D(is_regularization=True, S=r, gamma=cfg['metric_gamma']),
                    optimizer=torch.optim.Adam(model.parameters(), lr=cfg['lr']))
    n, S = case['batch'], case.get('nodes', 0)
    if kind == 'attn_layer':
        torch.manual_seed(seed)
        with torch.device('cuda'):
            layer = Sp_GalerkinAttention(HIDDEN, HEADS, POS, 1e-6, 0.0, 0.0, 1e-2, 1e-2, False).eval()
        return dict(kind=kind, layer=layer, x=torch.randn(n, S, HIDDEN, device='cuda', generator=g), position=_positions(n, S, g))
    if kind == 'attn_ops_grad':
        leaf = lambda ts: [t.requires_grad_() for t in ts]
        return dict(kind=kind, x=torch.randn(n, S, HIDDEN, device='cuda', generator=g).requires_grad_(), position=_positions(n, S, g),
                    q=leaf(_projection(g)[:2]), k=leaf(_projection(g)), v=leaf(_projection(g)),
                    grad=torch.randn(n, HEADS, S, POS + HEAD_DIM, device='cuda', generator=g))
    if kind == 'projpos':
        return dict(kind=kind, x=torch.randn(n, S, HIDDEN, device='cuda', generator=g), position=_positions(n, S, g), w=_projection(g))
    if kind == 'skinny':
        w = case['width']
        return dict(kind=kind, a=torch.randn(n, w, S, device='cuda', generator=g), b=torch.randn(n, S, w, device='cuda', generator=g),
                    alpha=1.0 / S)
    torch.manual_seed(seed)
    with torch.device('cuda'):
        layer = Sp_SpectralConv2D(HEAD_DIM, HEAD_DIM, case['modes'], 0.0, 'silu').eval()
    with torch.no_grad():
        for p in layer.fourier_weight:
            p.copy_(torch.rand(p.shape, device='cuda', generator=g) / HEAD_DIM ** 2)
    return dict(kind=kind, layer=layer, x=torch.randn(n, case['r'], case['r'], HEAD_DIM, device='cuda', generator=g))


# ------------------------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------------------------
def run(state):
    kind = state['kind']
    if kind == 'infer':
        with torch.no_grad():
            return state['model'](state['node'], state['position'], state['grid'])
    if kind == 'host':
        with torch.no_grad():
            return state['engine'].run(state['batches'])
    if kind == 'train':
        model = state['model']
        loss = train_epoch_darcy(model, [state['batch']], state['loss'], state['optimizer'], device='cuda')
        vector = torch.nn.utils.parameters_to_vector
        return dict(loss=loss, grads=vector(p.grad for p in model.parameters()), params=vector(p.detach() for p in model.parameters()))
    if kind == 'attn_layer':
        with torch.no_grad():
            return state['layer'](state['x'], state['x'], state['x'], state['position'])
    if kind == 'attn_ops_grad':
        x, pos = state['x'], state['position']
        q = multihead_projection_with_position_rrc_cuda(x, *state['q'], pos, HEADS, HEAD_DIM, POS)
        k, v = (multihead_projection_layernorm_with_position_rrc_cuda(x, *w, pos, 1e-6, HEADS, HEAD_DIM, POS) for w in (state['k'], state['v']))
        out = multihead_galerkin_attention_cccr_cuda(q, k, v)
        leaves = [x, *state['q'], *state['k'], *state['v']]
        return dict(out=out.detach(), grads=torch.autograd.grad(out, leaves, state['grad']))
    with torch.no_grad():
        if kind == 'projpos':
            return multihead_projection_layernorm_with_position_rrc_cuda(state['x'], *state['w'], state['position'], 1e-6, HEADS, HEAD_DIM, POS)
        if kind == 'skinny':
            return batched_skinny_gemm(state['a'], state['b'], state['alpha'])
        return state['layer'](state['x'])


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def _spectral_flops(r, m):
    """Residual linear map, real-to-complex transform to m x 2m kept modes, mixing, and back, per sample (truncated sums)."""
    return 2 * r * r * 32 * 32 + 2 * (2 * r * r * 32 * 2 * m + 8 * r * 32 * m * 2 * m) + 8 * 2 * m * m * 32 * 32


def _attention_flops(nodes):
    """Q, K, V projections, K^T V and Q (K^T V), per sample."""
    return 2 * nodes * 3 * HIDDEN * HIDDEN + 2 * 2 * nodes * HEADS * 34 * 34


def _model_work(case):
    """(bytes in and out, bytes of weights, flops) of one forward."""
    cfg = _config(case)
    (r, _), (mid, _), (ra, _), _, _ = cfg['resolution_size']
    m, S = case['modes'], ra * ra
    flops = 2 * r * r * 9 * 128 + 2 * mid * mid * 9 * (128 * 42 + 42 * 42 + 42 * 44) + 2 * mid * mid * 9 * 128 * 128
    flops += 6 * (_attention_flops(S) + 2 * S * 136 * 128 + 2 * 2 * S * 128 * 256)
    flops += 2 * mid * mid * 128 * 32 + 2 * _spectral_flops(r, m) + 2 * r * r * (32 * 128 + 128)
    weights = 9 * (128 + 128 * 42 + 42 * 42 + 42 * 44 + 128 * 128) + 6 * (3 * 128 * 128 + 136 * 128 + 2 * 128 * 256) + 130 * 32
    weights += 2 * (4 * m * m * 32 * 32 + 32 * 32) + 32 * 128 + 128
    return case['batch'] * 4 * (r * r * (1 + 2 + 1) + 2 * S), 4 * weights, case['batch'] * flops


def work(case):
    kind = case['kind']
    if kind in ('infer', 'host', 'train'):
        data, weights, flops = _model_work(case)
        if kind == 'infer':
            return dict(bytes=data + weights, flops=flops)
        if kind == 'host':
            return dict(bytes=case['batches'] * data + weights, flops=case['batches'] * flops)
        # forward, two products for every forward product in the backward pass; weights and both Adam moments read and written
        return dict(bytes=2 * data + 7 * weights, flops=3 * flops)
    n, S = case['batch'], case.get('nodes', 0)
    x, heads = n * S * HIDDEN * 4, n * S * HEADS * 34 * 4
    if kind == 'attn_layer':
        return dict(bytes=2 * x + n * S * 8 + 4 * (3 * 128 * 128 + 136 * 128), flops=n * (_attention_flops(S) + 2 * S * 136 * 128))
    if kind == 'attn_ops_grad':
        return dict(bytes=2 * x + 2 * heads + n * S * 8 + 2 * 4 * 3 * 128 * 128, flops=3 * n * _attention_flops(S))
    if kind == 'projpos':
        return dict(bytes=x + heads + n * S * 8 + 4 * 128 * 128, flops=2 * n * S * 128 * 128)
    if kind == 'skinny':
        w = case['width']
        return dict(bytes=4 * n * (2 * w * S + w * w), flops=2 * n * w * w * S)
    r, m = case['r'], case['modes']
    return dict(bytes=4 * (2 * n * r * r * 32 + 4 * m * m * 32 * 32 + 32 * 32), flops=n * _spectral_flops(r, m))


def tolerance(case):
    """Relative 2-norm differences between correct fp32 implementations: rounding of one contraction for the single ops, of
    the whole chain of layers for the model, of the backward chain (with the sums over all nodes) for gradients; Adam turns
    the sign of a gradient that is zero but for rounding into a full step of a single weight, hence the largest difference."""
    if case['kind'] in ('infer', 'host'):
        return {'rel': 2e-5}
    if case['kind'] == 'train':
        return {'rel': 1e-4, 'max': 0.3}
    if case['kind'] == 'attn_ops_grad':
        return {'rel': 2e-5}
    return {'rel': 1e-5}
