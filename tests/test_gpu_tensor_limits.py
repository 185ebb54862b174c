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
