"""The ramp filter and the Siddon projector at the edges of their tiles, against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tomo():
    import tomogpi_b200 as t

    return t


def _cfg(t, nx, ny, nz, nu, nv, views, pitch, mag=2.0):
    fod = 2.0 * max(nx, ny)
    return t.ConfigCT(fod=fod, fdd=mag * fod, projection_nb=views, u_detector_size=pitch * nu, v_detector_size=pitch * nv,
                      u_detector_pixel_nb=nu, v_detector_pixel_nb=nv, x_volume_size=float(nx), y_volume_size=float(ny),
                      z_volume_size=float(nz), x_volume_pixel_nb=nx, y_volume_pixel_nb=ny, z_volume_pixel_nb=nz)


@pytest.mark.parametrize("nu,nv,views", [(5, 3, 2), (31, 4, 3), (33, 7, 5), (127, 5, 7), (130, 2, 17), (257, 3, 11), (700, 1, 3)])
def test_ramp_filter_edges(tomo, nu, nv, views):
    """The ramp filter at the edges of its tiles (32 rows, 128 outputs, 32-pixel segments),
    against the same taps applied in double: 2 nu FP32 products per output, so well within
    1e-5. A NaN pixel reaches the outputs within its lags and no other."""
    import oracle

    cfg = _cfg(tomo, 16, 16, 16, nu, nv, views, 2.0)
    s = np.random.default_rng(nu).random(cfg.sinogram_shape, dtype=np.float32)
    with tomo.Context(cfg) as ctx:
        got = ctx.ramp_filter(torch.from_numpy(s).cuda()).cpu().numpy()
        ref = oracle.ramp_filter(cfg, s)
        assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
        s[0, 0, nu // 2] = np.nan
        bad = np.isnan(ctx.ramp_filter(torch.from_numpy(s).cuda()).cpu().numpy())
    half = int(np.floor(nu / 2 + 0.5))
    lag = np.arange(nu) - nu // 2  # output i takes taps[i - j + half], 0 <= i - j + half < 2 half
    assert np.array_equal(bad[0, 0], (lag >= -half) & (lag < half))
    assert not bad[0, 1:].any() and not bad[1:].any()


@pytest.mark.parametrize("nu,nv,views", [(20, 400, 16), (63, 100, 5), (64, 200, 150), (130, 2, 17), (300, 50, 40), (1000, 4, 40),
                                         (1600, 3, 2)])
def test_ramp_filter_in_place(tomo, nu, nv, views):
    """The output may be the input: bit-identical to the filter into another buffer, row by row
    (few rows, or overlapping buffers) as in tiles."""
    cfg = _cfg(tomo, 16, 16, 16, nu, nv, views, 2.0)
    s = torch.rand(cfg.sinogram_shape, device="cuda")
    with tomo.Context(cfg) as ctx:
        ref = ctx.ramp_filter(s)
        got = s.clone()
        assert ctx.ramp_filter(got, out=got) is got
        assert torch.equal(got, ref)


@pytest.mark.parametrize("spec", [(9, 7, 5, 11, 6, 5, 2.0), (40, 40, 12, 61, 43, 11, 1.3), (33, 33, 70, 40, 90, 9, 2.0)],
                         ids=lambda s: "x".join(map(str, s)))
def test_siddon_matches_oracle(tomo, spec):
    """The Siddon projector's walk ends where an axis leaves the volume: flat, odd and deep
    volumes, rays that miss or graze it. FP32 against the FP32 restatement."""
    import oracle

    cfg = _cfg(tomo, *spec)
    vol = np.random.default_rng(9).random(cfg.volume_shape, dtype=np.float32)
    with tomo.Context(cfg) as ctx:
        got = ctx.project("SIDDON", torch.from_numpy(vol).cuda()).cpu().numpy()
        assert ctx.errors() == 0
    ref = oracle.project(cfg, oracle.SIDDON, vol)
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
