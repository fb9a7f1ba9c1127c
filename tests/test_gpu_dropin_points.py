"""Drop-in injection and extraction with host arrays beside the number of points up to which the kernel
reads the values from mapped memory: bitwise against the points applied in order in float32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npoints", [1, 4095, 4096, 4097])
@pytest.mark.parametrize("inject", [True, False])
def test_host_points(npoints, inject):
    from wavefd_b200 import spacetime
    rng = np.random.default_rng(npoints)
    nt, ntr, ncell = 3, 37, 5000
    pts = np.zeros(npoints, spacetime.SOURCEPOINT32)
    pts["iu"], pts["ir"] = rng.integers(1, ncell + 1, npoints), rng.integers(1, ntr + 1, npoints)
    pts["c"] = rng.standard_normal(npoints)
    field = rng.standard_normal(ncell).astype(np.float32)
    data = rng.standard_normal((ntr, nt)).astype(np.float32)
    want_f, want_d = field.copy(), data.copy()
    parts = spacetime.source_blocking(pts, 4) if inject else spacetime.receiver_blocking(pts, 4)
    for p in parts:
        for iu, ir, c in p:
            if inject:
                want_f[iu - 1] += c * data[ir - 1, 1]
            else:
                want_d[ir - 1, 1] += c * field[iu - 1]
    if inject:
        spacetime.injectdata(field, parts, data, 2)
    else:
        spacetime.extractdata(data, field, 2, parts)
    assert np.array_equal(field, want_f) and np.array_equal(data, want_d)


@pytest.mark.parametrize("per", [63, 64, 65, 200])
@pytest.mark.parametrize("groups", [1, 3])
@pytest.mark.parametrize("inject", [True, False])
def test_host_points_of_one_location(per, groups, inject):
    """Beside the number of values that one thread reads from mapped memory."""
    from wavefd_b200 import spacetime
    rng = np.random.default_rng(per)
    nt, ntr, ncell, n = 3, 400, 900, groups * per
    pts = np.zeros(n, spacetime.SOURCEPOINT32)
    one = np.repeat(np.arange(1, groups + 1) * 7, per)
    pts["iu"], pts["ir"] = (one, rng.integers(1, ntr + 1, n)) if inject else (rng.integers(1, ncell + 1, n), one)
    pts["c"] = rng.standard_normal(n)
    field = rng.standard_normal(ncell).astype(np.float32)
    data = rng.standard_normal((ntr, nt)).astype(np.float32)
    want_f, want_d = field.copy(), data.copy()
    for iu, ir, c in pts:
        if inject:
            want_f[iu - 1] += c * data[ir - 1, 1]
        else:
            want_d[ir - 1, 1] += c * field[iu - 1]
    if inject:
        spacetime.injectdata(field, [pts], data, 2)
    else:
        spacetime.extractdata(data, field, 2, [pts])
    assert np.array_equal(field, want_f) and np.array_equal(data, want_d)
