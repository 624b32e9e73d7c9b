"""The MDL gradient where the Gram matrix has an odd side (an odd number of
frames, fewer than modes): the eigenvectors lie behind an odd number of
eigenvalues in one buffer and must still be aligned to their 16-byte elements.

Against central differences of the value, windows frozen, at the tolerances of
the even sizes: cosine >= 0.99, each component within 5 % of the norm."""
import numpy as np
import pytest

from test_gpu_adjoint import KINDS, _case, _get, _grad_metric, _handle, _perturbed, _set, _steps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import digholo_b200
    return digholo_b200.load()


@pytest.mark.parametrize("frames,independent", [(33, 0), (31, 1)])
def test_odd_frame_count(lib, frames, independent):
    hol = _case(frames)
    cfg = _perturbed(hol, 0)
    h, keep = _handle(lib, cfg, hol.frames)
    lib.digHoloConfigSetAutoAlignPolIndependence(h, independent)
    assert lib.digHoloB200FreezeWindow(h, 1) == 0
    g = _grad_metric(lib, h, 1)[0]
    steps = _steps(lib, h, cfg)
    entries = [(pol, k) for pol in (0, 1) for k in KINDS[:5]] + [(None, "waist")]
    ga, gf = [], []
    for pol, kind in entries:
        base, d = _get(lib, h, pol or 0, kind), 0.05 * steps[kind]
        vals = []
        for sign in (1, -1):
            _set(lib, h, pol or 0, kind, base + sign * d)
            vals.append(_grad_metric(lib, h, 1)[1])
        _set(lib, h, pol or 0, kind, base)
        gf.append((vals[0] - vals[1]) / (2 * d) * steps[kind])
        ga.append((g[0, 5] + g[1, 5] if pol is None else g[pol, KINDS.index(kind)]) * steps[kind])
    lib.digHoloDestroy(h)
    ga, gf = np.array(ga), np.array(gf)
    norm = np.linalg.norm(gf)
    assert ga @ gf / (np.linalg.norm(ga) * norm) >= 0.99
    assert np.abs(ga - gf).max() <= 0.05 * norm
