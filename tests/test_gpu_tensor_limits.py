"""The edges of the rule that leaves subgrids to the kernels without tensor cores."""
import numpy as np
import pytest
import torch

import idg_gb300._lib as L
from gpu_helpers import dev, spec_for

pytestmark = pytest.mark.gpu


def _general(S):
    """Launch shapes that take any geometry, as the library picks them."""
    g = 24 if S == 32 else 22 if 64 % (S // 2) == 0 else 11 if S == 24 else 12 if S == 48 else 13
    return g, 34 if S == 32 else 32 if S >= 32 and S % 8 == 0 else 31


def _both(S, run):
    """run() on the tensor-core shapes and on general ones."""
    from idg_gb300 import tuning

    saved, last = tuning.get_shapes(S), tuning.num_shapes()
    try:
        tuning.set_shapes(S, last[0] - 1, last[1] - 1)
        here = run()
        tuning.set_shapes(S, *_general(S))
        return here, run()
    finally:
        tuning.set_shapes(S, *saved)


def test_a_subgrid_too_long_for_the_bounded_waits_is_the_general_kernels(idg):
    """One subgrid of 2^23 + 64 visibilities: the same bits as the general kernel,
    which has no wait that lasts as long as a subgrid."""
    from idg_gb300 import ops

    S, C, T, G = 32, 64, (1 << 17) + 1, 512
    rng = np.random.default_rng(1)
    k = (2 * np.pi * np.linspace(150e6, 160e6, C) / 299792458.0).astype(np.float32)
    md = np.zeros(1, L.METADATA_DTYPE)
    md["nr_timesteps"], md["station2"], md["x"], md["y"] = T, 1, 240, 240
    uvw = dev((40.0 * rng.standard_normal((T, 3))).astype(np.float32))
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    vis = torch.view_as_complex(torch.randn(T, C, 4, 2, generator=g, device="cuda"))
    sub = torch.view_as_complex(torch.randn(1, 4, S, S, 2, generator=g, device="cuda"))
    at = torch.tensor([1, 0, 0, 1], dtype=torch.complex64, device="cuda").repeat(1, 2, S, S, 1).contiguous()
    sp, common = spec_for(G, S, C, 2, 1, 0.05), (dev(md), uvw, dev(k))
    taper = torch.ones(S, S, device="cuda")
    ops.device_status(clear=True)

    def grid():
        out = torch.empty_like(sub)
        ops.gridder(sp, *common, vis, taper, at, out, variant=L.VARIANT_BATCHED)
        return out.cpu().numpy()

    def degrid():
        out = torch.zeros_like(vis)
        ops.degridder(sp, *common, out, taper, at, sub, variant=L.VARIANT_BATCHED)
        return out.cpu().numpy()

    for run in (grid, degrid):
        here, general = _both(S, run)
        assert np.array_equal(here, general) and np.abs(here).max() > 0
    assert ops.device_status(clear=True) == 0


def _edge_case(S, image_size, limit, n=3000, C=3, T=4, G=512):
    """Subgrids of T rows whose range of w (or reach of u) steps through the
    limit, one unit in the last place of the larger end at a time."""
    step, edge = image_size / S, 0.5 * (S - 1) * image_size / S
    nn = lambda r2: 1 - np.sqrt(1 - r2)
    k = (2 * np.pi * np.linspace(150e6, 160e6, C) / 299792458.0).astype(np.float32)
    rng = np.random.default_rng(S)
    rows = np.zeros((n, T, 3), np.float32)
    rows[:, :, :2] = 40.0 * rng.standard_normal((n, T, 2))
    half = {"eps": 2e-3 / (2 * np.pi * (nn(2 * edge**2) - 2 * nn(edge**2))), "slope": 0.75 / nn(edge**2), "reach": 1.0}[limit]
    w = half * 2 * np.pi / 1.0001 / float(k[-1])  # range -w .. w, the largest wavenumber
    at = 65536.0 * 2 * np.pi / step / float(k[-1]) if limit == "reach" else w
    ends = (np.float32(at).view(np.int32) + np.arange(n, dtype=np.int32) - n // 2).view(np.float32)
    if limit == "reach":
        rows[:, 2, 0] = ends
    else:
        rows[:, 0, 2], rows[:, 1, 2] = -ends, ends
        rows[:, 2:, 2] = ends[:, None] * rng.uniform(-1, 1, (n, T - 2)).astype(np.float32)
    md = np.zeros(n, L.METADATA_DTYPE)
    md["time_offset"], md["nr_timesteps"], md["station2"] = T * np.arange(n), T, 1
    md["x"], md["y"] = rng.integers(0, G - S, (2, n))
    return spec_for(G, S, C, 2, 1, image_size), md, rows.reshape(-1, 3), k


@pytest.mark.parametrize("S", [10, 16, 24, 32, 48])
@pytest.mark.parametrize("image_size,limit", [(0.05, "slope"), (0.15, "eps"), (0.05, "reach")])
def test_every_subgrid_on_the_edge_of_the_rule_is_done_by_one_kernel(idg, S, image_size, limit):
    """Outputs start as NaN; both kernels take part, so the edge is inside the range."""
    from idg_gb300 import ops

    T = 64 if S < 16 else 8  # long enough for the tensor-core kernels
    sp, md, uvw, k = _edge_case(S, image_size, limit, T=T)
    n, C = len(md), len(k)
    g = torch.Generator(device="cuda")
    g.manual_seed(S)
    vis = torch.view_as_complex(torch.randn(T * n, C, 4, 2, generator=g, device="cuda"))
    sub = torch.view_as_complex(torch.randn(n, 4, S, S, 2, generator=g, device="cuda"))
    at = torch.tensor([1, 0, 0, 1], dtype=torch.complex64, device="cuda").repeat(1, 2, S, S, 1).contiguous()
    common, taper = (dev(md), dev(uvw), dev(k)), torch.ones(S, S, device="cuda")

    def grid():
        out = torch.full_like(sub, float("nan"))
        ops.gridder(sp, *common, vis, taper, at, out, variant=L.VARIANT_BATCHED)
        return out.reshape(n, -1).cpu().numpy()

    def degrid():
        out = torch.full_like(vis, float("nan"))
        ops.degridder(sp, *common, out, taper, at, sub, variant=L.VARIANT_BATCHED)
        return out.reshape(n, -1).cpu().numpy()

    for run in (grid, degrid):
        here, general = _both(S, run)
        assert np.isfinite(here).all(), f"{(~np.isfinite(here).all(axis=1)).sum()} subgrids done by neither kernel"
        same = (here == general).all(axis=1)
        assert same.any() and not same.all()


def test_a_wavenumber_that_is_not_a_number_is_the_general_kernels(idg):
    from idg_gb300 import ops

    S, n = 32, 3
    sp, md, uvw, k = _edge_case(S, 0.05, "slope", n=n)
    uvw[:, 2] = 10.0
    k[1] = np.nan
    rng = np.random.default_rng(3)
    vis = dev((rng.standard_normal((4 * n, 3, 4)) + 1j * rng.standard_normal((4 * n, 3, 4))).astype(np.complex64))
    at = torch.tensor([1, 0, 0, 1], dtype=torch.complex64, device="cuda").repeat(1, 2, S, S, 1).contiguous()
    sub = torch.ones((n, 4, S, S), dtype=torch.complex64, device="cuda")
    args = (sp, dev(md), dev(uvw), dev(k))

    def grid():
        out = torch.zeros_like(sub)
        ops.gridder(*args, vis, torch.ones(S, S, device="cuda"), at, out, variant=L.VARIANT_BATCHED)
        return out.cpu().numpy()

    def degrid():
        out = torch.zeros_like(vis)
        ops.degridder(*args, out, torch.ones(S, S, device="cuda"), at, sub, variant=L.VARIANT_BATCHED)
        return out.cpu().numpy()

    for run in (grid, degrid):
        here, general = _both(S, run)
        assert np.array_equal(here, general, equal_nan=True)


@pytest.mark.parametrize("S", [16, 24, 32, 48])
@pytest.mark.parametrize("faint", [1e-2, 1e-4, 1e-8, 1e-20])
def test_a_faint_correlation_keeps_its_own_precision(oracle_mod, idg, S, faint):
    """Correlations of very different magnitude, not mixed by the A-terms: each one by
    itself is as close to FP64 as all of them together otherwise are (2e-6: the
    split operands, sincos, expansion and sums of test_gpu_tensor.py)."""
    from conftest import check_rel
    from gpu_helpers import degrid_gpu, grid_gpu
    from test_gpu_tensor import TOL, _case

    c = _case(S, [50, 3, 17], 9, seed=S)
    at = np.zeros_like(c["at"])
    at[..., 0], at[..., 3] = c["at"][..., 0], c["at"][..., 3]
    scale = np.array([1.0, faint, faint**0.5, 30.0], np.float32)
    sp = spec_for(c["G"], S, 9, c["ns"], 1, c["img"])
    prm = oracle_mod.params(c["G"], S, 9, c["ns"], 3, c["img"])
    vis, sub = c["vis"] * scale, c["sub"] * scale[None, :, None, None]
    got = grid_gpu(sp, c["md"], c["uvw"], c["k"], vis, c["taper"], at, L.VARIANT_BATCHED)
    want = oracle_mod.gridder(prm, c["uvw"], c["k"], vis, c["taper"], at, c["md"])
    for p in range(4):
        check_rel(f"gridder S={S} correlation {p} of {scale[p]}", got[:, p], want[:, p], TOL)
    got = degrid_gpu(sp, c["md"], c["uvw"], c["k"], sub, c["taper"], at, 70, L.VARIANT_BATCHED)
    want = oracle_mod.degridder(prm, c["uvw"], c["k"], sub, c["taper"], at, c["md"], 70)
    for p in range(4):
        check_rel(f"degridder S={S} correlation {p} of {scale[p]}", got[..., p], want[..., p], TOL)


# (S, subgrids, steps, channels) on both sides of the lines: at S = 12 and 40 by
# length, at 16, 24 and 48 also by the number of subgrids, and on the edges
@pytest.mark.parametrize("S,n,T,C,grid_tc,degrid_tc", [
    (8, 100, 3, 1, True, False), (8, 500, 11, 1, False, False), (8, 500, 12, 1, True, False), (8, 40, 64, 1, True, True),
    (12, 600, 13, 1, False, False), (12, 600, 36, 1, True, True), (12, 50, 35, 1, True, False), (16, 100, 3, 1, True, False),
    (16, 500, 3, 8, True, False), (16, 500, 12, 8, True, True), (16, 900, 3, 1, True, True), (14, 900, 8, 1, True, True),
    (24, 3000, 15, 1, False, True), (24, 3000, 16, 1, True, True), (24, 900, 3, 1, True, True), (34, 4000, 27, 1, False, True),
    (40, 300, 3, 1, True, True), (40, 600, 11, 1, False, True), (40, 1000, 10, 2, True, True), (48, 3000, 7, 2, False, True), (48, 900, 3, 1, True, True),
    (56, 3000, 5, 1, False, True), (64, 3000, 1, 1, True, True), (32, 3000, 1, 1, True, True)])
def test_short_subgrids_go_to_the_faster_kernel(idg, S, n, T, C, grid_tc, degrid_tc):
    """Where the rule says so, the default shape gives the general kernel's bits."""
    from idg_gb300 import ops

    G, rng = 512, np.random.default_rng(S + n)
    k = (2 * np.pi * np.linspace(150e6, 160e6, C) / 299792458.0).astype(np.float32)
    md = np.zeros(n, L.METADATA_DTYPE)
    md["time_offset"], md["nr_timesteps"], md["station2"] = T * np.arange(n), T, 1
    md["x"], md["y"] = rng.integers(0, G - S, (2, n))
    uvw = dev((40.0 * rng.standard_normal((T * n, 3))).astype(np.float32))
    g = torch.Generator(device="cuda")
    g.manual_seed(S)
    vis = torch.view_as_complex(torch.randn(T * n, C, 4, 2, generator=g, device="cuda"))
    sub = torch.view_as_complex(torch.randn(n, 4, S, S, 2, generator=g, device="cuda"))
    at = torch.tensor([1, 0, 0, 1], dtype=torch.complex64, device="cuda").repeat(1, 2, S, S, 1).contiguous()
    sp, common, taper = spec_for(G, S, C, 2, 1, 0.05), (dev(md), uvw, dev(k)), torch.ones(S, S, device="cuda")

    def grid():
        return ops.gridder(sp, *common, vis, taper, at, torch.empty_like(sub), variant=L.VARIANT_BATCHED).cpu().numpy()

    def degrid():
        return ops.degridder(sp, *common, torch.empty_like(vis), taper, at, sub, variant=L.VARIANT_BATCHED).cpu().numpy()

    for run, tensor in ((grid, grid_tc), (degrid, degrid_tc)):
        here, general = _both(S, run)
        assert np.array_equal(here, general) != tensor
        assert np.linalg.norm(here - general) <= 4e-6 * np.linalg.norm(general)


@pytest.mark.parametrize("S,n", [(24, 400), (32, 153), (48, 100)])
def test_a_plans_work_list_is_taken_as_it_is(idg, S, n):
    """A plan's list is longest first and every subgrid in it once: the same bits as the
    separate steps, which take the subgrids in another order."""
    from idg_gb300 import ops
    from test_gpu_tensor import _case

    rng = np.random.default_rng(n)
    lengths = [int(x) for x in rng.choice([0, 1, 9, 40, 40, 200, 400], n)]
    lengths[3] = 40
    c = _case(S, lengths, 9, seed=n)
    rows = slice(int(c["md"]["time_offset"][3]), int(c["md"]["time_offset"][3]) + 40)
    c["uvw"][rows, 2] += (8000.0 * np.sin(np.arange(40))).astype(np.float32)  # left to the general kernel
    data = [dev(c[k]) for k in ("uvw", "k", "vis", "taper", "at")]
    grids = [torch.zeros((1, 4, c["G"], c["G"]), dtype=torch.complex64, device="cuda") for _ in range(2)]
    sp = spec_for(c["G"], S, 9, c["ns"], 1, c["img"])
    plan = ops.Plan(sp, c["md"], c["uvw"].shape[0])
    plan.grid(*data, grids[0])
    sub = torch.empty((n, 4, S, S), dtype=torch.complex64, device="cuda")
    ops.gridder(spec_for(c["G"], S, 9, c["ns"], 1, c["img"], flags=L.IDG_FLAG_NO_TAPER), dev(c["md"]), *data[:3], None,
                data[4], sub, variant=L.VARIANT_BATCHED)
    ops.subgrid_fft(sp, sub, 1, data[3])
    bins = ops.TileBins(sp, c["md"])
    bins.add(sub, grids[1])
    assert torch.equal(torch.view_as_real(grids[0]), torch.view_as_real(grids[1])) and grids[0].abs().max() > 0
    assert plan.status() == 0
    bins.close()
    plan.close()


@pytest.mark.parametrize("S", [16, 32, 48])
def test_edges_of_the_gridders_chunks(oracle_mod, idg, S):
    """A chunk holds 256 visibilities: one below, at and above one and two of them."""
    from test_gpu_tensor import TOL, _case, _degrid, _grid

    c = _case(S, [255, 256, 257, 512, 513], 1, seed=S)
    _grid(c, oracle_mod, f"S={S} chunk edges", TOL)
    _degrid(c, oracle_mod, f"S={S} chunk edges", TOL)


@pytest.mark.parametrize("chunk", [0, 1, 2, 3])
def test_every_chunk_has_a_scale_of_its_own(oracle_mod, idg, chunk):
    """Four chunks of very different magnitude, all but one of them zero: its own
    contribution is as exact as any."""
    from test_gpu_tensor import TOL, _case, _grid

    c = _case(32, [256], 4, seed=12)
    keep = np.zeros(256, np.float32)
    keep[64 * chunk:64 * chunk + 64] = 10.0 ** (6 * chunk - 9)
    c["vis"] *= keep[:, None, None]
    _grid(c, oracle_mod, f"chunk {chunk}", TOL)
