"""Edges of the scatter kernel's entries, which are pairs of pixels that are neighbours along the last axis: images one to
three pixels wide, pairs half outside of the image, few entries and many, taps that do not fill the last batch; and each
kind of result wanted alone."""
import ctypes

import pytest
import torch

import cases
from cases import Case, cabi_problem, make_inputs, run_cabi, run_oracle

pytestmark = pytest.mark.gpu

EDGES = [
    Case('one_wide', 2, False, 2, 64, 64, (9, 1), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.0),
    Case('two_wide', 2, False, 3, 64, 64, (7, 2), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 2.0),
    Case('odd_width', 2, False, 2, 128, 64, (11, 13), (5, 5), (1, 2), (2, 2), (1, 1), (), 1, 2, 1, True, 3.0),
    Case('far_offsets', 2, False, 1, 64, 64, (6, 5), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 0, True, 30.0),
    Case('whole_pixels', 2, False, 1, 64, 64, (12, 11), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 0, 1, True, 0.0),
    Case('seven_taps', 1, False, 2, 64, 64, (131,), (7,), (1,), (3,), (1,), (), 1, 1, 1, True, 2.0),
    Case('length_one', 1, False, 5, 64, 128, (1,), (3,), (1,), (1,), (1,), (), 1, 1, 1, True, 1.0),
    Case('thin_volume', 3, False, 1, 64, 64, (4, 5, 1), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.0),
    Case('odd_volume', 3, False, 1, 64, 64, (3, 7, 9), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 2.0),
    # volumes are taken in blocks of 4 x 4 x 8 positions: several tiles, blocks cut off on every side
    Case('cut_blocks', 3, False, 2, 64, 64, (6, 9, 19), (3, 2, 3), (1, 1, 2), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.5),
    Case('scattered_output', 2, True, 2, 64, 64, (9, 7), (4, 4), (2, 2), (1, 1), (1, 1), (0, 0), 1, 1, 1, True, 2.0),
]


def _device_inputs(case, dtype, seed):
    x, w, off, mask, bias, go = make_inputs(case, seed=seed)
    if off is not None:
        off = (off * 64).round() / 64 + 1 / 128   # exact in f32, never on a pixel: one-sided derivatives are not compared
    t = [None if v is None else v.float() for v in (x, w, off, mask, bias, go)]
    t = [v if v is None or i in (2, 3, 4) else v.to(dtype) for i, v in enumerate(t)]
    return t, [None if v is None else v.cuda() for v in t]


@pytest.mark.parametrize('case', EDGES, ids=[c.name for c in EDGES])
@pytest.mark.parametrize('dtype,tol', [(torch.float32, 1e-4), (torch.bfloat16, 2e-2), (torch.float16, 5e-3)],
                         ids=['f32', 'bf16', 'f16'])
def test_edges(case, dtype, tol):
    host, dev = _device_inputs(case, dtype, 81)
    ref = run_oracle(case, *(None if t is None else t.double() for t in host))
    cases.assert_parity(run_cabi(case, *dev, engine=2), ref, tol, case.name)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16], ids=['f32', 'bf16'])
def test_each_result_alone(dtype):
    """Only the scattered image, only the coordinate gradients: the same values as all together."""
    from tvdcn_b200 import cabi
    L = cabi.lib()
    case = EDGES[2]
    _, dev = _device_inputs(case, dtype, 82)
    x, w, off, mask, bias, go = dev
    both = run_cabi(case, *dev, engine=2)
    p = cabi_problem(case, x.dtype, torch.float32, 2)
    ws = torch.empty(L.tvdcn_b200_backward_workspace_bytes(ctypes.byref(p)), dtype=torch.uint8, device='cuda')
    ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    for want in ((1, 0, 0), (0, 1, 1), (0, 1, 0), (0, 0, 1)):
        out = [torch.full_like(t, float('nan')) if k else None for k, t in zip(want, (x, off, mask))]
        cabi.check(L.tvdcn_b200_deform_conv_backward(
            ctypes.byref(p), ptr(go), ptr(x), ptr(w), ptr(off), ptr(mask), ptr(out[0]), None, ptr(out[1]), ptr(out[2]), None,
            ptr(ws), ws.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        for a, r in zip(out, (both[1], both[3], both[4])):
            # sums of a few hundred f32 terms in another order (bf16: and rounded)
            assert a is None or cases.nerr(a, r) <= (1e-5 if dtype == torch.float32 else 8e-3)


def test_infinite_gradient_stays_with_its_pixels():
    """A position whose grad_output is infinite reaches the pixels that it samples and no others, least of all across the
    ends of image rows."""
    case = Case('inf_gradient', 2, False, 1, 64, 64, (10, 7), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5)
    _, dev = _device_inputs(case, torch.float32, 83)
    for col in (0, 6):
        go = dev[5].clone()
        go[0, :, 4, col] = float('inf')
        got = run_cabi(case, *dev[:5], go, engine=2)[1]
        ref = run_cabi(case, *dev[:5], go, engine=1)[1]
        hit = lambda t: (~torch.isfinite(t)).any(dim=1)
        assert hit(ref).any() and not hit(ref).all()
        assert torch.equal(hit(got), hit(ref))


LONE = [   # entries that lack a pixel: without offsets all of them, and at every edge of a narrow image
    Case('lone_1d', 1, False, 2, 64, 64, (37,), (3,), (1,), (1,), (1,), (), 1, 0, 1, True, 0.0),
    Case('lone_2d', 2, False, 2, 64, 64, (6, 7), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 0, 1, True, 0.0),
    Case('lone_3d', 3, False, 2, 64, 64, (3, 4, 5), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 0, 1, True, 0.0),
    Case('single_pixels', 1, False, 5, 64, 64, (1,), (3,), (1,), (1,), (1,), (), 1, 1, 1, True, 1.0),
    Case('single_pixel', 2, False, 1, 64, 64, (1, 1), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.0),
    Case('one_wide_volume', 3, False, 1, 64, 64, (4, 3, 1), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.0),
    Case('lone_T', 2, True, 2, 64, 64, (5, 4), (4, 4), (2, 2), (1, 1), (1, 1), (0, 0), 1, 0, 1, True, 0.0),
]


@pytest.mark.parametrize('case', LONE, ids=[c.name for c in LONE])
@pytest.mark.parametrize('dtype,tol', [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=['f32', 'bf16'])
def test_lone_pixels(case, dtype, tol):
    host, dev = _device_inputs(case, dtype, 86)
    ref = run_oracle(case, *(None if t is None else t.double() for t in host))
    cases.assert_parity(run_cabi(case, *dev, engine=2), ref, tol, case.name)


@pytest.mark.parametrize('case', LONE, ids=[c.name for c in LONE])
@pytest.mark.parametrize('at', [0, -1], ids=['first', 'last'])
@pytest.mark.parametrize('what', ['gradient', 'mask'])
def test_lone_pixels_take_nothing_that_is_not_finite(case, at, what):
    """What an infinite gradient (in the transposed forward call: input) or a mask that is NaN reaches, and no neighbour of it.  The
    mask's bits are all ones."""
    _, dev = _device_inputs(case, torch.float32, 87)
    dense = 0 if case.transposed else 5
    if what == 'gradient':
        dev[dense].flatten(2)[0 if at == 0 else -1, :, at] = float('inf')
    else:
        dev[3].view(torch.int32).flatten(2)[0 if at == 0 else -1, :, at] = -1
    got, ref = run_cabi(case, *dev, engine=2), run_cabi(case, *dev, engine=1)
    i = 0 if case.transposed else 1
    hit = lambda t: (~torch.isfinite(t)).any(dim=1)
    assert hit(ref[i]).any() and torch.equal(hit(got[i]), hit(ref[i]))


@pytest.mark.parametrize('length', [1466, 1494], ids=['1466_tiles', '1494_tiles'])
def test_volumes_of_one_unit_per_tile(length):
    """f32, around ten tiles per SM: every unit begins a tile."""
    case = Case('volume', 3, False, 1, 64, 64, (2, 8, 8 * length), (1, 1, 2), (1, 1, 1), (0, 0, 0), (1, 1, 1), (), 1, 1, 1, True, 1.0)
    _, dev = _device_inputs(case, torch.float32, 84)
    got, ref = run_cabi(case, *dev, engine=2), run_cabi(case, *dev, engine=1)
    for a, r in zip((got[1], got[3], got[4]), (ref[1], ref[3], ref[4])):
        assert cases.nerr(a, r) <= 1e-4


ODD_OFFSETS = [
    Case('odd_offsets_1d', 1, False, 2, 64, 64, (70,), (3,), (1,), (1,), (1,), (), 1, 1, 1, True, 1.0),
    Case('odd_offsets_2d', 2, False, 2, 64, 64, (9, 11), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.0),
    Case('odd_offsets_3d', 3, False, 1, 64, 64, (4, 5, 7), (3, 2, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.0),
    Case('odd_offsets_T', 2, True, 2, 64, 64, (6, 7), (4, 4), (2, 2), (1, 1), (1, 1), (0, 0), 1, 1, 1, True, 1.0),
]


@pytest.mark.parametrize('value', [float('inf'), float('-inf'), 1e30, float('nan')], ids=['inf', 'minus_inf', 'huge', 'nan'])
@pytest.mark.parametrize('case', ODD_OFFSETS, ids=[c.name for c in ODD_OFFSETS])
@pytest.mark.parametrize('dtype,aux,tol', [(torch.float32, torch.float32, 1e-4), (torch.bfloat16, torch.float32, 2e-2),
                                           (torch.float16, torch.float16, 5e-3)], ids=['f32', 'bf16', 'f16'])
def test_offsets_that_are_not_finite(case, dtype, aux, tol, value):
    """A cell outside of the image, however far, has no gradients; a NaN offset's are those of the SIMT kernels, value by value."""
    _, dev = _device_inputs(case, dtype, 85)
    dev = [t.to(aux) if i in (2, 3, 4) else t for i, t in enumerate(dev)]
    off = dev[2].flatten(2)
    for axis in range(case.dim):     # some positions of every (tap, axis), each axis at positions of its own
        off[:, axis::case.dim, axis::case.dim + 2] = value
    got, ref = run_cabi(case, *dev, engine=2), run_cabi(case, *dev, engine=1)
    if value == value:
        assert all(torch.isfinite(r).all() for r in ref)
        cases.assert_parity(got, ref, tol, case.name)
    for i in (3, 4) if case.transposed else (1, 3, 4):
        finite = torch.isfinite(ref[i])
        assert torch.equal(torch.isfinite(got[i]), finite), cases.NAMES[i]
        assert cases.nerr(torch.where(finite, got[i], 0), torch.where(finite, ref[i], 0)) <= tol, cases.NAMES[i]


@pytest.mark.parametrize('case', ODD_OFFSETS, ids=[c.name for c in ODD_OFFSETS])
def test_infinite_mask_of_a_cell_outside(case):
    """Its product with the zeros of a cell outside of the image is NaN, on both engines."""
    _, dev = _device_inputs(case, torch.float32, 88)
    dev[2].flatten(2)[:, 0, 3] = 1e30
    dev[3].flatten(2)[:, 0, 3] = float('inf')
    got, ref = run_cabi(case, *dev, engine=2)[3], run_cabi(case, *dev, engine=1)[3]
    assert torch.isnan(ref).any() and torch.equal(torch.isfinite(got), torch.isfinite(ref))
