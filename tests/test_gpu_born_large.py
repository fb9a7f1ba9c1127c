"""VEA Born injections and imaging conditions, 2D and 3D, fast build (whose TTI injection rotates back before
the divergence) against the strict build of the same calls (the reference's order, bitwise against the
restatement in the parity tests). Increments: relative L2 1e-5, the fast build's bound in the parity tests."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(9, 9, 9), (40, 33, 103), (64, 129, 132), (9, 9), (301, 64), (130, 257)]  # (nx[, ny], nz)


@pytest.mark.parametrize("physics", ["vti", "tti"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fs", [True, False])
def test_fast_born_vea(physics, shape, fs):
    import ctypes

    import torch
    from wavefd_b200 import props, synthetic
    from wavefd_b200.codec import _CAI
    variant, nd = "VEA", len(shape)
    cls = getattr(props, f"Prop{nd}DAco{physics.upper()}DenQ_DEO2_FDTD")
    size = dict(nx=shape[0], nz=shape[-1], dx=9.0, dz=10.0, **({"ny": shape[1], "dy": 12.0} if nd == 3 else {}))
    p = cls(nsponge=4, dt=0.0005, freesurface=fs, **size)
    arr = lambda k: torch.as_tensor(_CAI(ctypes.cast(getattr(p.abi, "get" + k)(p.p), ctypes.c_void_p).value, shape),  # noqa: E731
                                    device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    rnd = lambda s=1.0: torch.randn(shape, generator=gen, device="cuda") * s  # noqa: E731
    for k, t in synthetic.earth_model(shape if nd == 3 else (shape[0], 1, shape[1]), physics, seed=3, nsponge=4,
                                      device="cuda").items():
        if hasattr(p.abi, "get" + k):
            arr(k).copy_(t.reshape(shape))
    cur = ["PCur", "MCur"]
    for k in ["POld", "MOld"]:
        arr(k).copy_(rnd())
    wf = {k: rnd() for k in ("pold", "mold")}
    wf.update({k: rnd(50.0) for k in ("pspace", "mspace")})
    keys = ("v", "ϵ", "η")
    dm = {k: rnd({"v": 30.0, "b": 0.02}.get(k, 0.01)) for k in keys}
    mt = getattr(props, p.NAME + "_Model_" + variant)()
    got = []
    for strict in (True, False):
        p.set_strict(strict)
        for k in cur:
            arr(k).zero_()
        img = {k: torch.zeros(shape, device="cuda") for k in keys}
        torch.cuda.synchronize()
        props.forwardBornInjection(p, mt, dm, wf)
        props.adjointBornAccumulation(p, mt, props.ImagingConditionStandard(), img, wf)
        got.append([arr(k).clone() for k in cur] + list(img.values()))
    for a, b, k in zip(*got, cur + list(keys)):
        assert float(a.abs().max()) > 0
        err = float((a.double() - b.double()).norm() / a.double().norm())
        assert err <= 1e-5, f"{physics} {variant} {shape} fs={fs} {k}: {err:.2e}"
    props.free(p)
