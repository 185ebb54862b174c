"""The tensor-core gridder and degridder at the edges of their blocks, tiles and
chunks, on both sides of the rule that leaves subgrids to the general kernels,
and at magnitudes far from one.

Tolerance.  Against FP64 the split operands leave 2^-22 per factor, the two SFU
sincos of a phasor at most 5e-7 each, the neglected second order of the
expansion at most 1e-7 RMS and the fp32 sums and truncation 3e-7: 1.2e-6 in all
if every bound is met at once, so 2e-6.  Where the general kernel is the one
that runs, the repository's 1e-5.
"""
import numpy as np
import pytest

import idg_gb300._lib as L
from conftest import check_rel
from gpu_helpers import degrid_gpu, grid_gpu, spec_for

pytestmark = pytest.mark.gpu

TOL, TOL_GENERAL = 2e-6, 1e-5
C_LIGHT = 299792458.0


def _case(S, lengths, C, seed, w_metres=200.0, image_size=0.05, G=512, ns=5):
    """Subgrids of the given numbers of timesteps with random tracks that fit them;
    w_metres is the spread of w inside a subgrid."""
    rng = np.random.default_rng(seed)
    n, rows = len(lengths), int(sum(lengths))
    freqs = np.linspace(150e6, 160e6, C)
    k = (2 * np.pi * freqs / C_LIGHT).astype(np.float32)
    md = np.zeros(n, L.METADATA_DTYPE)
    md["time_offset"] = np.concatenate([[0], np.cumsum(lengths)[:-1]])
    md["nr_timesteps"] = lengths
    md["station1"] = rng.integers(0, ns - 1, n)
    md["station2"] = ns - 1
    md["x"] = rng.integers(0, G - S, n)
    md["y"] = rng.integers(0, G - S, n)
    of = np.repeat(np.arange(n), lengths)
    cells = 0.3 * S * (rng.random((rows, 2)) - 0.5)  # about the subgrid's centre
    centre = np.stack([md["x"][of] + S / 2 - G / 2, md["y"][of] + S / 2 - G / 2], 1)
    uv = (centre + cells) / image_size * C_LIGHT / 155e6
    w = (3000.0 * rng.standard_normal(n))[of] + w_metres * (rng.random(rows) - 0.5)
    uvw = np.concatenate([uv, w[:, None]], 1).astype(np.float32)
    at = (np.array([1, 0, 0, 1]) + 0.1 * (rng.standard_normal((1, ns, S, S, 4)) +
                                          1j * rng.standard_normal((1, ns, S, S, 4)))).astype(np.complex64)
    taper = (0.5 + rng.random((S, S))).astype(np.float32)
    vis = (rng.standard_normal((rows, C, 4)) + 1j * rng.standard_normal((rows, C, 4))).astype(np.complex64)
    sub = (rng.standard_normal((n, 4, S, S)) + 1j * rng.standard_normal((n, 4, S, S))).astype(np.complex64)
    return dict(S=S, G=G, C=C, ns=ns, img=image_size, md=md, uvw=uvw, k=k, at=at, taper=taper, vis=vis, sub=sub)


def _degrid(c, oracle_mod, name, tol, scale=1.0):
    sp = spec_for(c["G"], c["S"], c["C"], c["ns"], 1, c["img"])
    prm = oracle_mod.params(c["G"], c["S"], c["C"], c["ns"], len(c["md"]), c["img"])
    got = degrid_gpu(sp, c["md"], c["uvw"], c["k"], c["sub"] * np.float32(scale), c["taper"], c["at"],
                     c["uvw"].shape[0], L.VARIANT_BATCHED)
    want = oracle_mod.degridder(prm, c["uvw"], c["k"], c["sub"], c["taper"], c["at"], c["md"], c["uvw"].shape[0])
    check_rel(f"degridder {name}", got.astype(np.complex128) / np.float64(np.float32(scale)), want, tol)


def _grid(c, oracle_mod, name, tol, scale=1.0):
    sp = spec_for(c["G"], c["S"], c["C"], c["ns"], 1, c["img"])
    prm = oracle_mod.params(c["G"], c["S"], c["C"], c["ns"], len(c["md"]), c["img"])
    got = grid_gpu(sp, c["md"], c["uvw"], c["k"], c["vis"] * np.float32(scale), c["taper"], c["at"],
                   L.VARIANT_BATCHED)
    want = oracle_mod.gridder(prm, c["uvw"], c["k"], c["vis"], c["taper"], c["at"], c["md"])
    check_rel(f"gridder {name}", got.astype(np.complex128) / np.float64(np.float32(scale)), want, tol)


# lengths x channels: one visibility, and one below, at and above 16, 32, 128 and 256
EDGES = [([1, 2, 5], 3), ([16, 17, 31, 32, 33], 1), ([127, 128, 129], 1), ([8, 15, 17], 16), ([3], 100)]


@pytest.mark.parametrize("S", [8, 10, 16, 18, 24, 30, 32, 34, 48, 50, 64])
def test_degridder_block_and_tile_edges(oracle_mod, idg, S):
    for i, (lengths, C) in enumerate(EDGES):
        _degrid(_case(S, lengths, C, seed=100 * S + i), oracle_mod, f"S={S} {lengths}x{C}", TOL)


@pytest.mark.parametrize("subgrids", [1, 60, 151, 153])
def test_degridder_tiles_shared_out(oracle_mod, idg, subgrids):
    """Few subgrids: their tiles go to several CTAs."""
    _degrid(_case(24, [40] * subgrids, 10, seed=subgrids), oracle_mod, f"{subgrids} subgrids", TOL)


@pytest.mark.parametrize("S", [24, 48])
@pytest.mark.parametrize("subgrids", [153, 158])
def test_degridder_long_subgrids_shared_out(idg, S, subgrids):
    """Long subgrids are cut into segments that their neighbours' claims take.  A
    visibility's arithmetic does not depend on the cut, so the same subgrids in
    calls of a few (cut another way) give the same bits; one long subgrid is
    wider than the expansion holds for, and the last group is not full."""
    tiles = [1, 31, 32, 33, 48, 1, 1, 63, 64, 65, 80, 1, 200]
    lengths = [max(1, 8 * tiles[i % len(tiles)] + (i % 3) - 1) if i % 2 or i > 140 else 5 for i in range(subgrids)]
    c = _case(S, lengths, 16, seed=subgrids)
    long = int(np.argmax(np.asarray(lengths) > 400))
    rows = slice(int(c["md"]["time_offset"][long]), int(c["md"]["time_offset"][long]) + lengths[long])
    c["uvw"][rows, 2] += (8000.0 * np.sin(np.arange(lengths[long]))).astype(np.float32)
    sp = spec_for(c["G"], S, c["C"], c["ns"], 1, c["img"])

    def run(lo, hi):
        return degrid_gpu(sp, c["md"][lo:hi], c["uvw"], c["k"], c["sub"][lo:hi], c["taper"], c["at"],
                          c["uvw"].shape[0], L.VARIANT_BATCHED)

    whole = run(0, subgrids)
    assert np.all(np.abs(whole).sum(axis=2) > 0)
    parts = sum(run(lo, min(lo + 40, subgrids)) for lo in range(0, subgrids, 40))
    assert np.array_equal(whole, parts)


@pytest.mark.parametrize("S,subgrids", [(24, 160), (24, 161), (24, 191), (48, 45), (48, 64)])
@pytest.mark.parametrize("even", [False, True])
def test_gridder_longest_first(idg, S, subgrids, even):
    """More items than CTAs are taken by length.  A subgrid's sum does not depend on
    when it is taken, so calls of a few subgrids (in the plan's order) give the
    same bits; groups of 32 that are full, of one and of less, lengths with ties
    and zeros, and one subgrid that the expansion does not hold for."""
    rng = np.random.default_rng(subgrids)
    lengths = [20] * subgrids if even else [int(x) for x in rng.choice([0, 1, 7, 40, 40, 90, 300], subgrids)]
    if not even:
        lengths[3] = 40
    c = _case(S, lengths, 9, seed=subgrids)
    rows = slice(int(c["md"]["time_offset"][3]), int(c["md"]["time_offset"][3]) + lengths[3])
    c["uvw"][rows, 2] += (8000.0 * np.sin(np.arange(lengths[3]))).astype(np.float32)
    sp = spec_for(c["G"], S, c["C"], c["ns"], 1, c["img"])
    few = 30 if S > 32 else 120

    def run(lo, hi):
        return grid_gpu(sp, c["md"][lo:hi], c["uvw"], c["k"], c["vis"], c["taper"], c["at"], L.VARIANT_BATCHED)

    whole = run(0, subgrids)
    parts = np.concatenate([run(lo, min(lo + few, subgrids)) for lo in range(0, subgrids, few)])
    assert np.array_equal(whole, parts)
    assert all((np.abs(whole[i]).max() > 0) == (lengths[i] > 0) for i in range(subgrids))


def _wide(image_size):
    """Subgrids the expansion does not hold for, between others that it holds for."""
    c = _case(32, [40, 40, 40, 40], 8, seed=3, image_size=image_size)
    wide = np.repeat([False, True, False, True], 40)
    c["uvw"][wide, 2] += (8000.0 * np.sin(np.arange(wide.sum()))).astype(np.float32)
    return c


@pytest.mark.parametrize("image_size", [0.05, 0.2])
def test_degridder_wide_w(oracle_mod, idg, image_size):
    _degrid(_wide(image_size), oracle_mod, f"wide w, image {image_size}", TOL_GENERAL)


def _both(S, args, run, general, gridding):
    """The same call on the tensor-core shape and on a general one."""
    from idg_gb300 import tuning

    saved, last = tuning.get_shapes(S), tuning.num_shapes()
    try:
        tuning.set_shapes(S, *((last[0] - 1, saved[1]) if gridding else (saved[0], last[1] - 1)))
        here = run(*args)
        tuning.set_shapes(S, *((general, saved[1]) if gridding else (saved[0], general)))
        return here, run(*args)
    finally:
        tuning.set_shapes(S, *saved)


def test_degridder_image_too_wide_is_the_general_kernel(idg):
    c = _wide(0.5)
    sp = spec_for(c["G"], 32, 8, c["ns"], 1, c["img"])
    args = (sp, c["md"], c["uvw"], c["k"], c["sub"], c["taper"], c["at"], 160, L.VARIANT_BATCHED)
    here, general = _both(32, args, degrid_gpu, 34, False)
    assert np.array_equal(here, general)


@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-12, 1e12, 1e30])
def test_degridder_magnitudes(oracle_mod, idg, scale):
    c = _case(24, [20, 33], 7, seed=9)
    if scale == 0.0:
        sp = spec_for(c["G"], 24, 7, c["ns"], 1, c["img"])
        assert not degrid_gpu(sp, c["md"], c["uvw"], c["k"], 0 * c["sub"], c["taper"], c["at"], c["uvw"].shape[0],
                              L.VARIANT_BATCHED).any()
    else:
        _degrid(c, oracle_mod, f"scale {scale}", TOL, scale)


def test_degridder_values_that_are_not_finite(idg):
    """A NaN or infinity in a subgrid reaches its own visibilities and no others."""
    c = _case(32, [20, 20, 20], 4, seed=4)
    c["sub"][1, 2, 5, 7] = np.nan
    c["sub"][2, 0, 31, 0] = np.inf
    sp = spec_for(c["G"], 32, 4, c["ns"], 1, c["img"])
    got = degrid_gpu(sp, c["md"], c["uvw"], c["k"], c["sub"], c["taper"], c["at"], 60, L.VARIANT_BATCHED)
    assert np.isfinite(got[:20]).all()
    assert not np.isfinite(got[20:40]).all() and not np.isfinite(got[40:]).all()


@pytest.mark.parametrize("S", [16, 24, 32, 64])
def test_degridder_equals_the_general_kernel(idg, S):
    c = _case(S, [37, 64, 5], 9, seed=S)
    sp = spec_for(c["G"], S, 9, c["ns"], 1, c["img"])
    args = (sp, c["md"], c["uvw"], c["k"], c["sub"], c["taper"], c["at"], c["uvw"].shape[0], L.VARIANT_BATCHED)
    here, general = _both(S, args, degrid_gpu, 31, False)
    check_rel(f"degridder S={S} against the general kernel", here, general, TOL + 1e-6)


@pytest.mark.parametrize("S", [8, 10, 16, 18, 24, 30, 32, 34, 48, 50, 64])
def test_gridder_block_and_chunk_edges(oracle_mod, idg, S):
    for i, (lengths, C) in enumerate(EDGES):
        _grid(_case(S, lengths, C, seed=200 * S + i), oracle_mod, f"S={S} {lengths}x{C}", TOL)


@pytest.mark.parametrize("image_size", [0.05, 0.2])
def test_gridder_wide_w(oracle_mod, idg, image_size):
    _grid(_wide(image_size), oracle_mod, f"wide w, image {image_size}", TOL_GENERAL)


def test_gridder_image_too_wide_is_the_general_kernel(idg):
    c = _wide(0.5)
    sp = spec_for(c["G"], 32, 8, c["ns"], 1, c["img"])
    here, general = _both(32, (sp, c["md"], c["uvw"], c["k"], c["vis"], c["taper"], c["at"], L.VARIANT_BATCHED),
                          grid_gpu, 24, True)
    assert np.array_equal(here, general)


@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-12, 1e12, 1e30])
def test_gridder_magnitudes(oracle_mod, idg, scale):
    c = _case(24, [20, 33], 7, seed=9)
    if scale == 0.0:
        sp = spec_for(c["G"], 24, 7, c["ns"], 1, c["img"])
        assert not grid_gpu(sp, c["md"], c["uvw"], c["k"], 0 * c["vis"], c["taper"], c["at"], L.VARIANT_BATCHED).any()
    else:
        _grid(c, oracle_mod, f"scale {scale}", TOL, scale)


def test_gridder_chunks_of_very_different_magnitude(oracle_mod, idg):
    """Chunks of 128 visibilities carry scales of their own."""
    c = _case(32, [256], 4, seed=12)
    c["vis"] *= (10.0 ** np.linspace(-9, 9, 256)).astype(np.float32)[:, None, None]
    _grid(c, oracle_mod, "mixed magnitudes", TOL)


def test_gridder_values_that_are_not_finite(idg):
    """A NaN or infinity in a visibility reaches its own subgrid and no others."""
    c = _case(32, [20, 20, 20], 4, seed=4)
    c["vis"][25, 2, 1] = np.nan
    c["vis"][59, 0, 3] = np.inf
    sp = spec_for(c["G"], 32, 4, c["ns"], 1, c["img"])
    got = grid_gpu(sp, c["md"], c["uvw"], c["k"], c["vis"], c["taper"], c["at"], L.VARIANT_BATCHED)
    assert np.isfinite(got[0]).all() and not np.isfinite(got[1]).all() and not np.isfinite(got[2]).all()


@pytest.mark.parametrize("S", [16, 24, 32, 64])
def test_gridder_equals_the_general_kernel(idg, S):
    c = _case(S, [37, 64, 5], 9, seed=S)
    sp = spec_for(c["G"], S, 9, c["ns"], 1, c["img"])
    args = (sp, c["md"], c["uvw"], c["k"], c["vis"], c["taper"], c["at"], L.VARIANT_BATCHED)
    here, general = _both(S, args, grid_gpu, 13, True)
    check_rel(f"gridder S={S} against the general kernel", here, general, TOL + 1e-6)
