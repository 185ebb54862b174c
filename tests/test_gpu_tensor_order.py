"""Subgrids larger than 32 are degridded in four blocks, each adding to the
visibilities that the one before stored.  With an odd number of tiles of 128
visibilities a tile changes its result warpgroup from block to block, so the
sum holds only if a block's stores are waited for; with one tile nothing else
lies between them.  Pixels and visibilities are larger than the L2 cache.

Tolerance against a kernel without tensor cores, per visibility and relative to
the largest: 2^-22 per split factor, 5e-7 per sincos, 1e-5 in all; a lost block
is an error of the order of one.
"""
import numpy as np
import pytest
import torch

import idg_gb300._lib as L
from gpu_helpers import dev, spec_for
from test_gpu_tensor import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,subgrids,T", [(34, 4000, 8), (48, 2000, 8), (48, 2000, 3), (64, 1200, 8), (48, 700, 24),
                                          (64, 12, 8), (48, 9, 136)])
def test_degridder_blocks_add_in_order(idg, S, subgrids, T):
    """Repeated calls give the same bits, and every visibility has all four blocks.
    T of 16 channels: one tile, a part of one, three; few subgrids: their tiles in
    segments of one and of an odd number."""
    from idg_gb300 import ops, tuning

    c = _case(S, [T] * subgrids, 16, seed=S + T)
    sp = spec_for(c["G"], S, 16, c["ns"], 1, c["img"])
    vis = torch.zeros((T * subgrids, 16, 4), dtype=torch.complex64, device="cuda")
    args = (dev(c["md"]), dev(c["uvw"]), dev(c["k"]), vis, dev(c["taper"]), dev(c["at"]), dev(c["sub"]))

    def run():
        vis.fill_(float("nan"))
        ops.degridder(sp, *args, variant=L.VARIANT_BATCHED)
        torch.cuda.synchronize()
        return vis.clone()

    first = run()
    for _ in range(10):
        assert torch.equal(torch.view_as_real(run()), torch.view_as_real(first))
    saved = tuning.get_shapes(S)
    try:
        tuning.set_shapes(S, saved[0], 31)
        want = run()
    finally:
        tuning.set_shapes(S, *saved)
    assert float((first - want).abs().max() / want.abs().max()) <= 1e-5
