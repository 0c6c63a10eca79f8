"""Edges of how the tensor-core kernels share their work between CTAs: forward tiles that two CTAs sum together, CTAs that
walk several tiles (the next dense tile is loaded under the old one), remainders of the split, volumes with one CTA per
tile, and the line below which a padded transposed forward stays on the SIMT kernel."""
import json
import threading

import pytest
import torch

import cases
from cases import Case, make_inputs, nerr, run_cabi, run_oracle
from test_tensor_gpu import kernels_launched

pytestmark = pytest.mark.gpu

SPLITS = [
    # one tile, long reduction: two CTAs share it
    Case('one_long_tile', 2, False, 1, 256, 64, (9, 9), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 2, 1, True, 1.5),
    # three tiles of 27 chunks: two CTAs each, whose halves differ by a chunk
    Case('odd_halves', 2, False, 1, 192, 256, (17, 19), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    # 150 tiles: two of them over a full wave, shared ranges with pieces at both ends of a CTA
    Case('wave_plus_two', 2, False, 2, 128, 64, (98, 97), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 1, True, 1.5),
    # several tiles per CTA, two groups: tiles of one group follow those of the other
    Case('many_tiles_groups', 2, False, 2, 128, 128, (120, 107), (3, 1), (1, 1), (1, 0), (1, 1), (), 2, 2, 1, True, 2.0),
    # one tap and one chunk: a tile is a single unit everywhere
    Case('single_units', 2, False, 1, 64, 64, (150, 141), (1, 1), (1, 1), (0, 0), (1, 1), (), 1, 1, 1, True, 1.0),
    # dense channels that fill tensor memory (f32: one accumulator beside the dense tile)
    Case('one_accumulator', 2, False, 1, 64, 384, (130, 150), (3, 3), (1, 1), (1, 1), (1, 1), (), 1, 1, 0, True, 1.0),
]


@pytest.mark.parametrize('case', SPLITS, ids=[c.name for c in SPLITS])
@pytest.mark.parametrize('dtype,tol', [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)], ids=['f32', 'bf16'])
def test_split_work(case, dtype, tol):
    x, w, off, mask, bias, go = make_inputs(case, seed=71)
    # coordinates that f32 holds exactly: one that rounds across an integer has another derivative than in f64
    off = (off * 64).round() / 64 + 1 / 128
    q = lambda t, d: None if t is None else t.to(d)
    dev = (q(x, dtype), q(w, dtype), q(off, torch.float32), q(mask, torch.float32), q(bias, torch.float32), q(go, dtype))
    ref = run_oracle(case, *(None if t is None else t.double() for t in dev))
    dev = [None if t is None else t.cuda() for t in dev]
    got = run_cabi(case, *dev, engine=2)
    cases.assert_parity(got, ref, tol, case.name)
    # shared tiles are summed in a fixed order: the same call gives the same bits
    assert torch.equal(got[0], run_cabi(case, *dev, engine=2)[0])
    from tvdcn_b200 import cabi
    assert cabi.lib().tvdcn_b200_device_status() == 0


def test_dense_tile_is_reloaded_behind_the_last_mma_on_it():
    """384 dense channels of f32 leave tensor memory for one accumulator, 153 tiles give a few CTAs two: the second dense
    tile may overwrite the first only behind its last MMA, whatever the timing of the call."""
    case = SPLITS[-1]
    dev = [None if t is None else t.float().cuda() for t in make_inputs(case, seed=75)]
    ref = run_cabi(case, *dev, engine=1)
    for _ in range(25):
        cases.assert_parity(run_cabi(case, *dev, engine=2)[:2], ref[:2], 1e-4, case.name)


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16], ids=['f32', 'bf16'])
def test_last_tile_of_a_cta_is_read_behind_its_last_mma(dtype):
    """One tap and one chunk: a CTA's second tile is sampled while the first is summed, and its result may be read only
    when its own sums are complete, whatever the timing: the same bits from every call."""
    case = Case('two_units', 2, False, 4, 64, 64, (150, 41), (1, 1), (1, 1), (0, 0), (1, 1), (), 1, 1, 1, True, 1.0)
    dev = [t.float().cuda() for t in make_inputs(case, seed=76)]
    dev = [dev[0].to(dtype), dev[1].to(dtype), *dev[2:5], dev[5].to(dtype)]
    ref = run_cabi(case, *dev, engine=1)[0]
    first = run_cabi(case, *dev, engine=2)[0]
    assert nerr(first, ref) <= (1e-4 if dtype == torch.float32 else 2e-2)
    for _ in range(25):
        assert torch.equal(run_cabi(case, *dev, engine=2)[0], first)


def test_shared_tiles_of_calls_that_overlap():
    """Two host threads on two streams through tiles that CTAs share: partial sums and arrival counters are each call's own,
    so every call gives the bits of the same call alone."""
    from tvdcn_b200 import ops
    jobs = []
    for case in (SPLITS[0], SPLITS[1]):      # one tile of 36 chunks; three of 27
        x, w, off, mask, bias, _ = (t.float().cuda() for t in make_inputs(case, seed=78))
        jobs.append((torch.cuda.Stream(), lambda a=(x, w, off, mask, bias): ops.deform_conv2d(*a, padding=1)))
    want = [job() for _, job in jobs]
    torch.cuda.synchronize()
    results = [[], []]

    def work(i):
        with torch.cuda.stream(jobs[i][0]):
            results[i] = [jobs[i][1]() for _ in range(40)]
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for one, many in zip(want, results):
        assert len(many) == 40 and all(torch.equal(one, r) for r in many)


def scatter_grids(fn, path):
    """Runs fn() under the profiler; returns (numbers of CTAs of the scatter kernel's launches, fn's result)."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = fn()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    events = json.loads(path.read_text())['traceEvents']
    return [e['args']['grid'][0] for e in events if 'dcn_dgrad_tc' in e.get('name', '') and 'grid' in e.get('args', {})], out


@pytest.mark.parametrize('width,kernel,ctas', [
    (59, (3, 3, 3), 148), (60, (3, 3, 3), 1487),      # 1463 and 1487 tiles of nine units
    (60, (1, 2, 3), 148), (60, (1, 7, 1), 1487),      # two and three units per tile
], ids=['few_tiles', 'many_tiles', 'two_units', 'three_units'])
def test_volume_with_one_cta_per_tile(width, kernel, ctas, tmp_path):
    """f32: as many CTAs as tiles from 1480 tiles of at least three units on, else one per SM.  Too large for the CPU oracle, so the
    SIMT kernels, which are checked against it elsewhere, stand in."""
    pad = tuple(k // 2 for k in kernel)
    extent = tuple(n + k - 1 - 2 * p for n, k, p in zip((26, 61, width), kernel, pad))     # of the input: 26 x 61 x width positions
    case = Case('volume', 3, False, 2, 64, 64, extent, kernel, (1, 1, 1), pad, (1, 1, 1), (), 1, 1, 1, True, 1.0)
    dev = [t.float().cuda() for t in make_inputs(case, seed=72)]
    grids, got = scatter_grids(lambda: run_cabi(case, *dev, engine=2), tmp_path / 'trace.json')
    assert grids in ([ctas], [])       # (none where the profiler cannot see kernels)
    cases.assert_parity(got, run_cabi(case, *dev, engine=1), 1e-4, case.name)


@pytest.mark.parametrize('width', [58, 60], ids=['290_tiles', '300_tiles'])
def test_volume_of_16_bit_data(width):
    """Around two tiles per SM."""
    case = Case('volume16', 3, False, 1, 64, 64, (16, 40, width), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), (), 1, 1, 1, True, 1.0)
    x, w, off, mask, bias, go = (t.float().cuda() for t in make_inputs(case, seed=77))
    dev = [x.bfloat16(), w.bfloat16(), off, mask, bias, go.bfloat16()]
    cases.assert_parity(run_cabi(case, *dev, engine=2), run_cabi(case, *dev, engine=1), 2e-2, case.name)


@pytest.mark.parametrize('batch,simt', [(148, True), (149, False)], ids=['one_wave', 'more'])
def test_small_padded_transposed_forward_stays_simt(batch, simt):
    case = Case('tiny_T', 1, True, batch, 8, 16, (64,), (4,), (2,), (1,), (1,), (), 1, 1, 1, True, 1.5)
    dev = [t.float() for t in make_inputs(case, seed=73)]
    ref = run_oracle(case, *(t.double() for t in dev))
    dev = [t.cuda() for t in dev]
    names, got = kernels_launched(lambda: run_cabi(case, *dev))
    assert (names.get('gemm_scatter', 0) == 1) == simt, names
    cases.assert_parity(got, ref, 1e-5, case.name)
