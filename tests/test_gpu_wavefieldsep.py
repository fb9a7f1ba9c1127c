"""The wavefield-separation imaging condition at the edges of its transform lengths, against float64
FFTs of the zero-padded columns (the definition, not the kernel's closed form).

The kernel picks the power of two >= nz as its transform length (16 to 8192), so the depths here sit on
and beside those powers. Tolerance: a cell passes three transforms (operator, forward, inverse) of at
most 5 stages with about 4 roundings each, 60 roundings of 2^-24 taken at their worst.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 60 * 2.0 ** -24


def _expected(fields, V, B, isfwi):
    acc = 0.0
    for x, y in fields:
        nz = x.shape[-1]
        n = 2 * nz
        parts = []
        for f, cut in ((x, slice(nz + 1, n)), (y, slice(1, nz) if isfwi else slice(nz + 1, n))):
            s = np.fft.ifft(f.astype(np.float64), n=n, axis=-1)
            s[..., cut] = 0
            parts.append(np.fft.fft(s, axis=-1)[..., :nz])
        acc = acc + (parts[0] * parts[1]).real
    return 2 * B.astype(np.float64) / V.astype(np.float64) ** 3 * acc


@pytest.mark.parametrize("physics,ndim", [("iso", 2), ("tti", 3)])
@pytest.mark.parametrize("nz", [9, 15, 16, 17, 31, 33, 64, 65, 129, 251, 256, 257, 400, 511, 512, 513, 1000, 1025, 2049,
                                4096, 8192])
def test_every_transform_length(nz, physics, ndim):
    import torch
    from wavefd_b200 import props
    if ndim == 3 and nz > 1100:
        pytest.skip("the 2D object covers the deepest columns")
    cls = props.Prop2DAcoIsoDenQ_DEO2_FDTD if physics == "iso" else props.Prop3DAcoTTIDenQ_DEO2_FDTD
    shape = (11, nz) if ndim == 2 else (9, 13, nz)
    p = cls(nz=nz, nx=shape[0], nsponge=4, **({"ny": shape[1]} if ndim == 3 else {}))
    rng = np.random.default_rng(nz)
    f = lambda: rng.standard_normal(shape).astype(np.float32)  # noqa: E731
    V = (1500 + 3000 * rng.random(shape)).astype(np.float32)
    B = (0.5 + rng.random(shape)).astype(np.float32)
    # amplitudes as far apart as a V^2/B-scaled derivative and a pressure can be, and per field
    saved, old = [np.float32(a) * f() for a in (3e5, 2e-3)], [np.float32(a) * f() for a in (1e-6, 40.0)]
    props.V(p)[...], props.B(p)[...], props.POld(p)[...] = V, B, old[0]
    if physics == "tti":
        props.MOld(p)[...] = old[1]
    p.prefetch()
    mt = getattr(props, p.NAME + "_Model_V")()
    wf = {"pspace": torch.from_numpy(saved[0]).cuda(), "mspace": torch.from_numpy(saved[1]).cuda()}
    torch.cuda.synchronize()
    pairs = list(zip(saved, old))[: 1 if physics == "iso" else 2]
    for isfwi, cond in ((1, props.ImagingConditionWaveFieldSeparationFWI()),
                        (0, props.ImagingConditionWaveFieldSeparationRTM())):
        img = torch.zeros(shape, device="cuda")
        torch.cuda.synchronize()
        props.adjointBornAccumulation(p, mt, cond, {"v": img}, wf)
        want = _expected(pairs, V, B, isfwi)
        err = np.linalg.norm(img.cpu().numpy() - want) / np.linalg.norm(want)
        assert err <= TOL, f"nz={nz} isfwi={isfwi}: rel L2 {err:.2e}"
    props.free(p)
