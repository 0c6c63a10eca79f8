"""Shapes and types that reach the tensor-core kernels by padding or widening: channels per group off the multiples of
64, 16-bit offset / mask / bias, rows of the dense tensor that TMA cannot read (spatial extent off the multiples of 8).
They must run there (ENGINE_TENSOR) and keep the precision of f32 columns: the tolerances are far inside those of the
unpadded shapes (f32 data) or half a unit of the 16-bit results."""
import os
import subprocess
import sys

import pytest
import torch

import cases
from cases import Case, make_inputs, run_cabi, run_oracle
from test_tensor_gpu import kernels_launched

pytestmark = pytest.mark.gpu

SHAPES = [
    # name, dim, transposed, batch, cin, cout, size, kernel, stride, padding, dilation, outpad, groups, og, mg, bias, std
    Case('c8', 2, False, 2, 8, 8, (9, 11), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('c40_72_odd', 2, False, 3, 40, 72, (11, 9), (3, 3), (2, 1), (1, 1), (1, 1), (), 1, 1, 0, True, 2.0),
    Case('uneven_groups', 2, False, 2, 48, 80, (8, 9), (3, 2), (1, 1), (1, 0), (1, 2), (), 2, 3, 1, True, 1.5),
    Case('c65_odd_extent', 2, False, 2, 65, 130, (7, 7), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, False, 1.0),
    Case('c200_many_columns', 2, False, 1, 200, 256, (13, 12), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('c64_pitch', 2, False, 2, 64, 64, (7, 9), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('1d', 1, False, 3, 24, 16, (203,), (5,), (1,), (4,), (2,), (), 1, 1, 1, True, 3.0),
    Case('3d', 3, False, 2, 32, 32, (4, 5, 7), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.0),
    Case('T2d', 2, True, 2, 24, 40, (7, 6), (4, 4), (2, 2), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('T2d_groups', 2, True, 2, 48, 32, (5, 9), (3, 3), (2, 2), (1, 1), (1, 1), (1, 1), 2, 4, 2, True, 1.5),
    Case('7x7_taps', 2, False, 1, 16, 24, (10, 9), (7, 7), (1, 1), (3, 3), (1, 1), (), 1, 1, 1, True, 1.5),
]


@pytest.mark.parametrize('case', SHAPES, ids=[c.name for c in SHAPES])
@pytest.mark.parametrize('dtype,aux,tol', [
    (torch.float32, torch.float32, 5e-6), (torch.bfloat16, torch.float32, 4.5e-3),
    (torch.bfloat16, torch.bfloat16, 4.5e-3), (torch.float16, torch.float16, 6e-4)],
    ids=['f32', 'bf16', 'bf16_aux16', 'f16_aux16'])
def test_padded_and_widened_shapes(case, dtype, aux, tol):
    x, w, off, mask, bias, go = make_inputs(case, seed=61)
    q = lambda t, d: None if t is None else t.to(d)
    dev = (q(x, dtype), q(w, dtype), q(off, aux), q(mask, aux), q(bias, aux), q(go, dtype))
    ref = run_oracle(case, *(None if t is None else t.double() for t in dev))
    names, got = kernels_launched(lambda: run_cabi(case, *(None if t is None else t.cuda() for t in dev), engine=2))
    assert not {'sample_gemm', 'gemm_scatter', 'sample_wgrad'} & set(names), names
    assert names.get('dcn_wgrad_tc', 0) == 1 and names.get('dcn_dgrad_tc', 0) >= 1, names
    if case.name == 'c64_pitch' and aux == torch.float32:
        # only the weight gradient is widened: the other kernels take this shape with two-part or 16-bit columns
        tol = 2e-5 if dtype == torch.float32 else 2e-2
    if case.name == '1d' and dtype == torch.float32:
        tol = 2e-5   # an f32 coordinate near 200 resolves 1.5e-5 pixels
    cases.assert_parity(got, ref, tol, case.name)
    from tvdcn_b200 import cabi
    assert cabi.lib().tvdcn_b200_device_status() == 0


def test_padded_call_without_room_for_its_workspace_runs_on_the_simt_kernels():
    """8 channels are padded to 64: the workspace of the tensor-core kernels is many times the tensors, and a program that
    has no room for it must not fail for that.  A shape that needs no padding still raises.  In a process of its own, whose
    allocator holds nothing else."""
    run = subprocess.run([sys.executable, '-c', 'import test_wide_shapes_gpu as t; t.padded_call_without_room()'],
                         cwd=os.path.dirname(__file__), capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-3000:]


def padded_call_without_room():
    from tvdcn_b200 import ops
    dev = lambda *s: torch.randn(*s, device='cuda')
    leaves = [dev(4, 8, 512, 512), dev(8, 8, 3, 3), dev(4, 18, 512, 512), torch.rand(4, 9, 512, 512, device='cuda'), dev(8)]
    for t in leaves:
        t.requires_grad_(True)
    plain = [dev(4, 64, 512, 512), dev(64, 64, 3, 3), dev(4, 18, 128, 128)]     # workspace 268 MB, output 17 MB
    grad = dev(4, 8, 512, 512)

    def step():
        out = ops.deform_conv2d(*leaves, padding=1)
        return (out.detach(), *torch.autograd.grad(out, leaves, grad))
    names, want = kernels_launched(step)
    assert names.get('dcn_fwd_tc', 0) == 1 and names.get('dcn_dgrad_tc', 0) == 1, names
    want = [t.cpu() for t in want]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.memory_reserved() + (240 << 20)     # outputs and gradients 190 MB, workspaces 268 and 590 MB
    try:
        torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
        names, got = kernels_launched(step)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            ops.deform_conv2d(*plain, stride=4, padding=1)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert names.get('sample_gemm', 0) == 1 and names.get('gemm_scatter', 0) == 1 and names.get('sample_wgrad', 0) == 1, names
    cases.assert_parity(got, want, 2e-5)


@pytest.mark.parametrize('scales', [
    # image, mask, weight, grad_output, bias: columns up to 16 x 60000, past f16's 65504 ...
    (15000., 16., 1e-3, 1e-3, 100.),
    # ... and columns near 1e-6, whose second part lies below f16's smallest step
    (1e-3, 1e-3, 1000., 100., 1e-3),
], ids=['large_columns', 'small_columns'])
@pytest.mark.parametrize('aux', [torch.float16, torch.float32], ids=['aux16', 'aux32'])
@pytest.mark.parametrize('case', [
    Case('padded', 2, False, 2, 40, 72, (17, 19), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('groups', 2, False, 2, 48, 80, (8, 9), (3, 2), (1, 1), (1, 0), (1, 2), (), 2, 3, 2, True, 1.5),
    # with f32 offsets only the weight gradient of this one is wide (an odd extent)
    Case('odd_extent', 2, False, 2, 64, 64, (7, 9), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    Case('transposed', 2, True, 2, 24, 40, (9, 10), (4, 4), (2, 2), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
], ids=lambda c: c.name)
def test_f16_columns_outside_the_range_of_f16(case, aux, scales):
    """The columns of the wide f16 mode are scaled into the range of their f16 parts: sums of large and of small ones are
    as exact as those of the SIMT kernels, which keep columns in f32 (half a unit of the f16 results)."""
    if case.name == 'odd_extent' and aux == torch.float32:
        pytest.skip('its forward keeps columns in f16, as the reference does')
    x, w, off, mask, bias, go = make_inputs(case, seed=62)
    sx, sm, sw, sg, sb = scales
    x, w, go = x.clamp(-4, 4), w * w.shape[1] ** 0.5, go.clamp(-3, 3)
    if case.transposed:   # the sampled image is grad_output, whose sum has to fit f16 as well
        x, go, sm = x * sg, go * sx / 100, sm * 100
    else:
        x, go = x * sx, go * sg
    dev = (x.half(), (w * sw).half(), off.to(aux), (mask * sm).to(aux), (bias * sb).to(aux), go.half())
    ref = run_oracle(case, *(t.double() for t in dev))
    assert all(float(r.abs().max()) < 65504 for r in ref), [float(r.abs().max()) for r in ref]
    names, got = kernels_launched(lambda: run_cabi(case, *(t.cuda() for t in dev), engine=2))
    assert not {'sample_gemm', 'gemm_scatter', 'sample_wgrad'} & set(names), names
    cases.assert_parity(got, ref, 6e-4, case.name)
