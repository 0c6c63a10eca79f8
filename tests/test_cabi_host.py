"""CPU-only checks of the C ABI: the library loads, exports what the header declares, and its host-side
logic (validation, output extents, workspace sizing) behaves.  No kernel is launched."""
import ctypes
import os
import re

import pytest

import cases
from tvdcn_b200 import cabi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, 'include', 'tvdcn_b200.h')).read()
    return sorted(set(re.findall(r'\b(tvdcn_b200_[a-z0-9_]+)\s*\(', text)))


def test_library_exports_every_declared_symbol():
    L = cabi.lib()
    names = declared_symbols()
    assert len(names) >= 12
    for n in names:
        assert hasattr(L, n), f'{n} declared in include/tvdcn_b200.h but not exported'


def test_version_and_arch():
    L = cabi.lib()
    assert L.tvdcn_b200_cuda_version() >= 12000
    assert L.tvdcn_b200_cuda_arch_flags().decode() == 'sm_100a'
    assert isinstance(L.tvdcn_b200_launch_count(), int)


def test_struct_layout_matches_header():
    # 4 int32 + 3 int64 + 6 int64 + 15 int32 + 4 int32
    assert ctypes.sizeof(cabi.Problem) == 168  # 164 bytes of fields, padded to the int64 alignment


@pytest.mark.parametrize('dim,tr', [(1, False), (2, False), (3, False), (1, True), (2, True), (3, True)])
def test_output_extent(dim, tr):
    c = cases.reference_fixture(dim, tr)
    p = cases.cabi_problem(c, __import__('torch').float32)
    assert tuple(p.out_size[a] for a in range(dim)) == c.out_size
    assert all(p.out_size[a] == 1 for a in range(dim, 3))


def test_config_extents():
    # deform_conv2d N=128 256->256 28x28 k3 p1 and deform_conv_transpose2d 32x32 -> 64x64 k4 s2 p1
    p = cabi.make_problem(2, False, cabi.F32, 128, 256, 256, (28, 28), (3, 3), (1, 1), (1, 1), (1, 1), 1, 4, 1)
    assert (p.out_size[0], p.out_size[1]) == (28, 28)
    p = cabi.make_problem(2, True, cabi.F32, 64, 256, 128, (32, 32), (4, 4), (2, 2), (1, 1), (1, 1), 1, 2, 1)
    assert (p.out_size[0], p.out_size[1]) == (64, 64)
    p = cabi.make_problem(1, False, cabi.F32, 64, 512, 512, (4096,), (5,), (1,), (4,), (2,), 8, 8, 1)
    assert p.out_size[0] == 4096


@pytest.mark.parametrize('kw,msg', [
    (dict(dim=4), 'dim'),
    (dict(groups=3), 'divisible by groups'),
    (dict(offset_groups=3), 'offset_groups'),
    (dict(mask_groups=3), 'mask_groups'),
    (dict(stride=(0, 1)), 'stride'),
    (dict(in_size=(1, 1), kernel=(3, 3), padding=(0, 0)), 'too small'),
    (dict(dtype=cabi.F64, aux_dtype=cabi.F32), 'aux_dtype'),
])
def test_invalid_problems_are_rejected(kw, msg):
    base = dict(dim=2, transposed=False, dtype=cabi.F32, batch=2, in_channels=4, out_channels=4, in_size=(8, 8),
                kernel=(3, 3), stride=(1, 1), padding=(1, 1), dilation=(1, 1), groups=1, offset_groups=2,
                mask_groups=1)
    base.update(kw)
    with pytest.raises(cabi.TvdcnError) as e:
        cabi.make_problem(**base)
    assert msg in str(e.value)


def test_workspace_sizes():
    L = cabi.lib()
    simt = dict(engine=cabi.ENGINE_SIMT)
    p32 = cabi.make_problem(2, False, cabi.F32, 2, 8, 8, (8, 8), (3, 3), (1, 1), (1, 1), (1, 1), 1, 1, 1, **simt)
    assert L.tvdcn_b200_forward_workspace_bytes(ctypes.byref(p32)) == 0
    assert L.tvdcn_b200_backward_workspace_bytes(ctypes.byref(p32)) == 0
    p16 = cabi.make_problem(2, False, cabi.BF16, 2, 8, 8, (8, 8), (3, 3), (1, 1), (1, 1), (1, 1), 1, 1, 1, **simt)
    # f32 accumulators for grad_input, grad_weight, grad_offset, grad_mask
    need = 2 * 8 * 64 * 4 + 8 * 8 * 9 * 4 + 2 * 18 * 64 * 4 + 2 * 9 * 64 * 4
    got = L.tvdcn_b200_backward_workspace_bytes(ctypes.byref(p16))
    assert need <= got <= need + 4 * 256
    assert L.tvdcn_b200_engine_name(ctypes.byref(p32), 0).decode() == 'simt'


def test_problems_too_large_for_the_tensor_kernels_are_planned_on_the_simt_ones():
    """The tensor-core launchers count their work in 32 bits and their grids in 16: a plan must not choose them beyond."""
    L = cabi.lib()

    def engine(*args, **kw):
        return L.tvdcn_b200_engine_name(ctypes.byref(cabi.make_problem(*args, **kw)), 0).decode()
    # sample -> GEMM: 129604 position tiles x (channels / 256) x 512 taps
    conv = lambda cout: engine(2, False, cabi.BF16, 1, 64, cout, (4096, 4096), (16, 32), (1, 1), (0, 0), (1, 1), 1, 0, 0,
                               aux_dtype=cabi.F32)
    assert conv(8192) == 'tcgen05' and conv(8448) == 'simt'
    # GEMM -> scatter: 131072 position tiles x (channels / 64) x 128 batches of four taps
    transposed = lambda cout: engine(1, True, cabi.BF16, 1, 64, cout, (1 << 24,), (512,), (1,), ((1 << 23) - 50000,), (1,), 1,
                                     0, 0, aux_dtype=cabi.F32)
    assert transposed(8128) == 'tcgen05' and transposed(8192) == 'simt'

    # weight gradient: a split for every 42 chunks of one image each, at most 65535; the 16-bit parts of grad_output, 3 KB
    # per image, are what the workspace no longer holds
    def backward_bytes(batch):
        p = cabi.make_problem(2, False, cabi.F32, batch, 64, 64, (1, 1), (1, 1), (1, 1), (0, 0), (1, 1), 1, 0, 0)
        return L.tvdcn_b200_backward_workspace_bytes(ctypes.byref(p))
    assert backward_bytes(2_700_000) > 2_700_000 * 3072 and backward_bytes(3_000_000) < 3_000_000 * 3072


@pytest.mark.parametrize('dim,transposed,dtype,cin,cout,positions,taps,backward,engine', [
    # one tap: up to 16 of 64 sampled channels, up to 64 dense ones
    (2, False, 'F32', 16, 64, 1024, 1, 0, 'simt'), (2, False, 'BF16', 16, 16, 1024, 1, 0, 'simt'),
    (2, False, 'F32', 17, 16, 1024, 1, 0, 'tcgen05'), (2, False, 'F32', 16, 72, 1024, 1, 0, 'tcgen05'),
    (2, False, 'F32', 16, 64, 1024, 9, 0, 'tcgen05'), (2, False, 'F32', 16, 64, 1024, 1, 1, 'tcgen05'),
    # 1-d f32: 8 and 9 channels; backward only above 32768 positions
    (1, False, 'F32', 9, 32, 1024, 5, 0, 'simt'), (1, False, 'F32', 10, 32, 1024, 5, 0, 'tcgen05'),
    (1, False, 'F32', 8, 40, 1024, 5, 0, 'tcgen05'), (1, False, 'BF16', 8, 8, 1024, 5, 0, 'tcgen05'),
    (1, False, 'F32', 8, 8, 32768, 5, 1, 'tcgen05'), (1, False, 'F32', 8, 8, 32769, 5, 1, 'simt'),
    # transposed forward: 8 to 10 sampled channels above 4096 (f32) or 65536 positions
    (2, True, 'F32', 8, 10, 4096, 16, 0, 'tcgen05'), (2, True, 'F32', 8, 10, 4225, 16, 0, 'simt'),
    (2, True, 'F32', 8, 11, 4225, 16, 0, 'tcgen05'), (2, True, 'F32', 72, 8, 4225, 16, 0, 'tcgen05'),
    (2, True, 'BF16', 8, 8, 65536, 16, 0, 'tcgen05'), (2, True, 'BF16', 8, 8, 66049, 16, 0, 'simt'),
    (2, True, 'F32', 8, 9, 33124, 16, 1, 'simt'), (2, True, 'F32', 8, 10, 33124, 16, 1, 'tcgen05'),
    (1, True, 'F32', 8, 8, 40000, 4, 1, 'tcgen05'),
    # transposed 1-d f32 forward within one wave of SIMT blocks
    (1, True, 'F32', 16, 16, 64 * 148, 4, 0, 'simt'), (1, True, 'F32', 16, 16, 64 * 148 + 1, 4, 0, 'tcgen05'),
    (1, True, 'F32', 17, 16, 330, 4, 0, 'tcgen05'), (1, True, 'BF16', 8, 16, 330, 4, 0, 'tcgen05'),
    (2, True, 'F32', 8, 16, 324, 16, 0, 'tcgen05'),
    # fewer than eight channels: never; not padded at all: always on the tensor cores
    (2, False, 'F32', 7, 64, 1024, 9, 0, 'simt'), (1, True, 'F32', 64, 64, 64, 4, 0, 'tcgen05'),
])
def test_lines_between_the_engines(dim, transposed, dtype, cin, cout, positions, taps, backward, engine):
    L = cabi.lib()
    side = positions if dim == 1 else round(positions ** 0.5)
    k = taps if dim == 1 else round(taps ** 0.5)
    stride, pad = (2, (k - 2) // 2) if transposed else (1, k // 2)
    p = cabi.make_problem(dim, transposed, getattr(cabi, dtype), 1, cin, cout, (side,) * dim, (k,) * dim, (stride,) * dim,
                          (pad,) * dim, (1,) * dim, 1, 1, 1, aux_dtype=cabi.F32)
    assert L.tvdcn_b200_engine_name(ctypes.byref(p), backward).decode() == engine
    if engine == 'simt' and min(cin, cout) >= 8:    # asked for, the tensor cores still take it
        p.engine = cabi.ENGINE_TENSOR
        assert L.tvdcn_b200_engine_name(ctypes.byref(p), backward).decode() == 'tcgen05'


def test_transposed_forward_needs_its_accumulator_and_weights_only():
    """Packed weights and the f32 accumulator of the output, nothing behind them: exactly the scratch that is built in."""
    L = cabi.lib()
    L.tvdcn_b200_static_scratch_bytes.restype = ctypes.c_size_t
    p = cabi.make_problem(2, True, cabi.F32, 1, 64, 64, (126, 128), (4, 4), (2, 2), (1, 1), (1, 1), 1, 1, 1)
    need = 2 * 64 * 64 * 16 * 2 + 252 * 256 * 64 * 4
    assert L.tvdcn_b200_forward_workspace_bytes(ctypes.byref(p)) == need == L.tvdcn_b200_static_scratch_bytes()


@pytest.mark.parametrize('transposed', [False, True])
@pytest.mark.parametrize('dtype', [cabi.F32, cabi.BF16])
def test_workspace_sizes_of_an_empty_batch(transposed, dtype):
    L = cabi.lib()
    p = cabi.make_problem(2, transposed, dtype, 0, 64, 64, (8, 8), (3, 3), (1, 1), (1, 1), (1, 1), 1, 1, 1)
    one = cabi.make_problem(2, transposed, dtype, 1, 64, 64, (8, 8), (3, 3), (1, 1), (1, 1), (1, 1), 1, 1, 1)
    for size in (L.tvdcn_b200_forward_workspace_bytes, L.tvdcn_b200_backward_workspace_bytes):
        assert 0 <= size(ctypes.byref(p)) < size(ctypes.byref(one))


def test_null_pointer_is_an_error_not_a_crash():
    L = cabi.lib()
    p = cabi.make_problem(2, False, cabi.F32, 2, 8, 8, (8, 8), (3, 3), (1, 1), (1, 1), (1, 1), 1, 0, 0)
    rc = L.tvdcn_b200_deform_conv_forward(ctypes.byref(p), None, None, None, None, None, None, None, 0, None)
    assert rc == 1 and b'NULL' in L.tvdcn_b200_last_error()
