"""The strips of the uv-grid FFT: every length (each has its own strip width
and pass sequence) and several w-planes, against the definition in FP64 at the
image of a few cells.  The cells sit on the edges of the strips, in the centre
and in the corners; the result is compared in every plane at rows and columns
next to the same edges.  Relative RMS <= 2e-6, as for the dense comparison:
the sum has as many roundings as there are passes.
"""
import numpy as np
import pytest
import torch

from conftest import check_rel
from gpu_helpers import spec_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,planes", [(64, 1), (64, 3), (128, 2), (256, 1), (512, 3), (1024, 2), (2048, 2), (4096, 1),
                                      (8192, 1)])
def test_strips(idg, G, planes):
    from idg_gb300 import ops

    rng = np.random.default_rng(G + planes)
    edges = np.array([0, 1, 2, 3, 15, 16, 31, 32, G // 2 - 1, G // 2, G // 2 + 1, G - 33, G - 4, G - 2, G - 1])
    corr = (1.0 + 0.2 * rng.standard_normal(G)).astype(np.float32)
    sp = spec_for(G, 32, 16, 4, 1, 0.05)
    sp.nr_w_planes = planes
    n = 24
    cells = np.stack([rng.integers(0, planes * 4, n), rng.choice(edges, n), rng.choice(edges, n)])
    values = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    at = np.sort(np.concatenate([edges, rng.integers(0, G, 9)]))
    d = torch.empty((planes, 4, G, G), dtype=torch.complex64, device="cuda")
    x = torch.from_numpy(at).cuda()
    for direction in (-1, 1):
        d.zero_()
        flat = d.view(planes * 4, G, G)
        want = np.zeros((planes * 4, at.size, at.size), np.complex128)
        for p, v, u, a in zip(*cells, values):
            flat[p, v, u] += complex(a)
            a = complex(a) * (float(corr[v]) * float(corr[u]) if direction > 0 else 1.0)
            ey = np.exp(direction * 2j * np.pi * (((v - G // 2) * (at - G // 2)) % G) / G)
            ex = np.exp(direction * 2j * np.pi * (((u - G // 2) * (at - G // 2)) % G) / G)
            want[p] += a * np.outer(ey, ex)
        if direction < 0:
            want *= np.outer(corr[at].astype(np.float64), corr[at].astype(np.float64))
        ops.grid_fft(sp, d, direction, torch.from_numpy(corr).cuda())
        got = flat[:, x][:, :, x].cpu().numpy()
        check_rel(f"grid fft strips G={G} planes={planes} dir={direction}", got, want, 2e-6)
