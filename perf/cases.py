"""Performance cases: what a program that uses this package asks of it, from one small inference call to the
largest training step of its benchmark configurations.

A case is one deformable convolution, plain or transposed, in 1, 2 or 3 dimensions, called through
``tvdcn_b200.ops``: the forward call alone under ``no_grad`` (inference), or the forward call and the gradients of
everything it was given (training).  Keys:

  dim, transposed       which operator
  train                 forward + backward, else forward
  dtype                 type of input, weight and output: float32, bfloat16 or float16
  aux                   type of offset, mask and bias: float32 (what autocast passes), or that of the input (a model
                        that was converted as a whole, ``model.half()``)
  batch, cin, cout, s0, s1, s2          sizes; s0 is the slowest spatial axis, unused axes are 1
  kernel, stride, padding, dilation     the same along every axis; outpad is the transposed output_padding
  groups, og, mg        convolution, offset and mask groups; mg = 0: no mask (the first version of the operator)
  softmax               the mask is mask_softmax over the taps of given logits
  sigma                 standard deviation of the offsets, in pixels
"""
import math

import torch

from tvdcn_b200 import ops

_CONV = {(1, False): ops.deform_conv1d, (2, False): ops.deform_conv2d, (3, False): ops.deform_conv3d,
         (1, True): ops.deform_conv_transpose1d, (2, True): ops.deform_conv_transpose2d,
         (3, True): ops.deform_conv_transpose3d}
_SOFTMAX = {1: ops.mask_softmax1d, 2: ops.mask_softmax2d, 3: ops.mask_softmax3d}
_BYTES = {'float32': 4, 'bfloat16': 2, 'float16': 2}


def _case(name=None, dim=2, transposed=False, train=True, dtype='float32', aux='float32', batch=1, cin=64, cout=64,
          size=(28, 28), kernel=3, stride=1, padding=1, dilation=1, outpad=0, groups=1, og=1, mg=1, softmax=False,
          sigma=2.0):
    size = tuple(size) + (1,) * (3 - dim)
    c = dict(dim=dim, transposed=transposed, train=train, dtype=dtype, aux=aux, batch=batch, cin=cin, cout=cout,
             s0=size[0], s1=size[1], s2=size[2], kernel=kernel, stride=stride, padding=padding, dilation=dilation,
             outpad=outpad, groups=groups, og=og, mg=mg, softmax=softmax, sigma=sigma)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # one image through one layer of a small network in 16 bits: the call a real-time program makes,
        # where the time is launches and host work
        _case('infer_2d_one_image', train=False, dtype='bfloat16', cin=64, cout=64, size=(28, 28)),
        # a detector's feature map, odd height and width, batch 1, the whole model converted to half precision
        _case('infer_2d_half_model', train=False, dtype='float16', aux='float16', cin=256, cout=256, size=(67, 101)),
        # a decoder that doubles the resolution of a few images under autocast, odd sizes
        _case('infer_transpose2d_decoder', transposed=True, train=False, dtype='bfloat16', batch=8, cin=128, cout=64,
              size=(45, 61), kernel=4, stride=2, sigma=1.5),
        # the smallest training step of the benchmark configurations
        _case('train_2d_small', batch=4, size=(56, 56), sigma=1.5),
        # channel counts that fit no tile, stride 2, ragged extent, without a mask
        _case('train_2d_odd_channels', batch=8, cin=40, cout=72, size=(33, 47), stride=2, mg=0),
        # the layer that halves the resolution in a late stage of a residual network, mixed precision, no mask
        _case('train_2d_downsample', dtype='bfloat16', batch=16, cin=256, cout=512, size=(27, 27), stride=2, mg=0),
        # a short clip through a narrow 3-d layer, mixed precision
        _case('train_3d_narrow', dim=3, dtype='bfloat16', batch=2, cin=32, cout=32, size=(5, 23, 31), sigma=1.0),
        # the residual-network stage the headline benchmark is quoted on, in both of its precisions
        _case('train_2d_stage_mixed', dtype='bfloat16', batch=128, cin=256, cout=256, og=4, mg=4, softmax=True),
        _case('train_2d_stage', batch=128, cin=256, cout=256, og=4, mg=4, softmax=True),
        # long sequences, grouped and dilated
        _case('train_1d_grouped', dim=1, batch=64, cin=512, cout=512, size=(4096,), kernel=5, padding=4, dilation=2,
              groups=8, og=8, mg=8, sigma=3.0),
        # volumes, 27 taps
        _case('train_3d_volume', dim=3, batch=8, size=(16, 56, 56), sigma=1.0),
        # the decoder's training step
        _case('train_transpose2d', transposed=True, batch=64, cin=256, cout=128, size=(32, 32), kernel=4, stride=2,
              og=2, mg=2, sigma=1.5),
    ]


def _grid(c, at_input):
    """Spatial extent of the input, or of the output."""
    size = [c['s0'], c['s1'], c['s2']][:c['dim']]
    if at_input:
        return size
    k, s, p, d = c['kernel'], c['stride'], c['padding'], c['dilation']
    if c['transposed']:
        return [(n - 1) * s - 2 * p + d * (k - 1) + 1 + c['outpad'] for n in size]
    return [(n + 2 * p - d * (k - 1) - 1) // s + 1 for n in size]


def _shapes(c):
    """Shapes of everything a case reads and writes."""
    taps = c['kernel'] ** c['dim']
    n, src, dst = c['batch'], _grid(c, True), _grid(c, False)
    where = src if c['transposed'] else dst  # offsets and masks lie on the dense side's grid
    ker = [c['kernel']] * c['dim']
    weight = [c['cin'], c['cout'] // c['groups']] if c['transposed'] else [c['cout'], c['cin'] // c['groups']]
    return dict(input=[n, c['cin']] + src, weight=weight + ker, offset=[n, c['og'] * taps * c['dim']] + where,
                mask=[n, c['mg'] * taps] + where if c['mg'] else None, bias=[c['cout']],
                output=[n, c['cout']] + dst)


def work(case):
    s = _shapes(case)
    size = {k: math.prod(v) if v else 0 for k, v in s.items()}
    data, aux = _BYTES[case['dtype']], _BYTES[case['aux']]
    given = data * (size['input'] + size['weight']) + aux * (size['offset'] + size['mask'] + size['bias'])
    # forward: what is given and the output; backward: grad_output, and a gradient for all that was given
    total = given + data * size['output']
    if case['train']:
        total += data * size['output'] + given
    dense = size['input'] // case['cin'] if case['transposed'] else size['output'] // case['cout']
    gemm = 2 * dense * case['cout'] * case['cin'] // case['groups'] * case['kernel'] ** case['dim']
    return {'bytes': total, 'flops': gemm * (3 if case['train'] else 1)}


def tolerance(case):
    # relative error of sums of products: 32-bit ones, or of values rounded to 16 bits
    return {'rel': 2e-5} if case['dtype'] == 'float32' else {'rel': 1e-2}


def _cost(c):
    w = work(c)
    # channel counts off the tiles of the matrix units weigh more, and so does a small launch's share of 27 taps
    odd = any(v % 64 for v in (c['cin'] // c['groups'], c['cout'] // c['groups'], c['cin'] // c['og']))
    return max(w['bytes'], w['flops'] / 50) * (24 if odd or c['aux'] != 'float32' else 1)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = max(max(w['bytes'], w['flops'] / 50) for w in map(work, listed()))
    while True:
        dim = rng.choices((1, 2, 3), (1, 4, 1))[0]
        transposed = rng.random() < 0.25
        dtype = rng.choice(('float32', 'bfloat16', 'float16'))
        aux = dtype if rng.random() < 0.25 else 'float32'
        if rng.random() < 0.75:   # the usual widths, and the groups that go with them
            cin, cout = (64 * rng.choice((1, 1, 2, 3, 4, 4, 6, 8)) for _ in range(2))
            most = math.gcd(cin // 64, cout // 64)
            groups = rng.choice([n for n in (1, 2, 4, 8) if most % n == 0]) if rng.random() < 0.25 else 1
            side = (cout if transposed else cin) // 64
            og, mg = (rng.choice([n for n in (1, 2, 4, 8) if side % n == 0 and (cin // 64) % n == 0])
                      for _ in range(2))
        else:
            cin, cout = (8 * _log(rng, 1, 25) for _ in range(2))
            groups, og, mg = 1, 1, 1
        if rng.random() < 0.3:
            mg = 0
        if transposed:
            kernel, stride, padding = rng.choice(((4, 2, 1), (3, 2, 1), (2, 2, 0), (3, 1, 1)))
            outpad, dilation = (1, 1) if (kernel, stride) == (3, 2) else (0, 1)
        else:
            kernel = rng.choice((3, 5, 7)) if dim == 1 else rng.choices((1, 3, 5), (1, 8, 1))[0] if dim == 2 else 3
            dilation = rng.choice((1, 1, 1, 2))
            padding, stride, outpad = dilation * (kernel - 1) // 2, rng.choice((1, 1, 1, 2)), 0
        if dim == 1:
            size = (_log(rng, 100, 8000),)
        elif dim == 2:
            h = _log(rng, 7, 160)
            size = (h, max(7, int(h * rng.uniform(0.7, 1.6))))
        else:
            h = _log(rng, 7, 60)
            size = (_log(rng, 4, 20), h, max(7, int(h * rng.uniform(0.7, 1.6))))
        c = _case(dim=dim, transposed=transposed, train=rng.random() < 0.6, dtype=dtype, aux=aux,
                  batch=_log(rng, 1, 128), cin=cin, cout=cout, size=size, kernel=kernel, stride=stride,
                  padding=padding, dilation=dilation, outpad=outpad, groups=groups, og=og, mg=mg,
                  softmax=mg > 0 and rng.random() < 0.3, sigma=round(rng.uniform(0.5, 3.0), 2))
        if _cost(c) <= top:
            return c


def prepare(case, seed):
    gen = torch.Generator(device='cuda').manual_seed(int(seed))
    s = _shapes(case)
    data, aux = getattr(torch, case['dtype']), getattr(torch, case['aux'])

    def normal(shape, sigma=1.0):
        return torch.empty(shape, device='cuda', dtype=torch.float32).normal_(0.0, sigma, generator=gen)

    bound = 1 / math.sqrt(math.prod(s['weight'][1:]))
    weight = torch.empty(s['weight'], device='cuda').uniform_(-bound, bound, generator=gen)
    t = {'input': normal(s['input']).to(data), 'weight': weight.to(data),
         'offset': normal(s['offset'], case['sigma']).to(aux), 'mask': None, 'bias': normal(s['bias'], 0.1).to(aux)}
    if s['mask']:
        mask = normal(s['mask']) if case['softmax'] else torch.rand(s['mask'], device='cuda', generator=gen)
        t['mask'] = mask.to(aux)
    state = {'case': case, 'tensors': t, 'grad': None}
    if case['train']:
        state['grad'] = normal(s['output']).to(data)
        for v in t.values():
            if v is not None:
                v.requires_grad_(True)
    return state


def _forward(c, t):
    mask = t['mask']
    if mask is not None and c['softmax']:
        mask = _SOFTMAX[c['dim']](mask, (c['kernel'],) * c['dim'])
    conv = _CONV[c['dim'], c['transposed']]
    args = [(c[k],) * c['dim'] for k in ('stride', 'padding')]
    if c['transposed']:
        args.append((c['outpad'],) * c['dim'])
    return conv(t['input'], t['weight'], t['offset'], mask, t['bias'], *args, (c['dilation'],) * c['dim'],
                c['groups'])


def run(state):
    c, t = state['case'], state['tensors']
    if not c['train']:
        with torch.no_grad():
            return {'output': _forward(c, t)}
    out = _forward(c, t)
    names = [k for k, v in t.items() if v is not None]
    grads = torch.autograd.grad(out, [t[k] for k in names], state['grad'])
    return dict({'output': out.detach()}, **{'grad_' + k: v for k, v in zip(names, grads)})
