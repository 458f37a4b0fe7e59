"""The forms staged in shared memory by TMA that the default tuning runs: the RS projector
(csrc/rs_stage.cuh; where the geometry allows it, as set_staging("fits") asks for here) and the VI and FDK backprojectors (csrc/vi_tma.cu), against
the forms that read global memory."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tomo():
    import tomogpi_b200 as t

    return t


def _cfg(t, nx, ny, nz, nu, nv, views, pitch, mag=2.0, fod=None):
    fod = 2.0 * max(nx, ny) if fod is None else fod
    return t.ConfigCT(fod=fod, fdd=mag * fod, projection_nb=views, u_detector_size=pitch * nu, v_detector_size=pitch * nv,
                      u_detector_pixel_nb=nu, v_detector_pixel_nb=nv, x_volume_size=float(nx), y_volume_size=float(ny),
                      z_volume_size=float(nz), x_volume_pixel_nb=nx, y_volume_pixel_nb=ny, z_volume_pixel_nb=nz)


# (nx, ny, nz, nu, nv, views, pitch, mag[, fod]): one partial tile; odd sizes with several
# tiles and chunks; unequal sides; pixels finer than a voxel; windows of the largest width and
# height; too wide to stage (the texture runs); a source close enough that rays leave their
# tile's axis; every pitch of the copies modulo 4
RS = [(9, 7, 5, 11, 6, 5, 2.0), (101, 83, 66, 131, 95, 13, 1.9), (64, 120, 40, 97, 33, 9, 2.0),
      (90, 90, 90, 300, 270, 7, 0.7), (120, 120, 120, 104, 108, 11, 2.4), (64, 64, 64, 20, 20, 9, 8.0),
      (80, 80, 80, 128, 128, 12, 3.5, 2.5, 60.0), (62, 63, 61, 65, 64, 16, 2.0)]


@pytest.mark.parametrize("kind", ["RS", "RS_UM"])
@pytest.mark.parametrize("spec", RS, ids=lambda s: "x".join(map(str, s)))
def test_staged_projection_equals_padded(tomo, spec, kind):
    """Same texels, same arithmetic: bit-identical to the padded layout, in FP32 and with a
    16-bit result; a volume of ones gives every ray its sample count in either form."""
    cfg = _cfg(tomo, *spec)
    vol = torch.from_numpy(np.random.default_rng(3).random(cfg.volume_shape, dtype=np.float32) + 0.25).cuda()
    with tomo.Context(cfg) as ctx:
        ctx.set_staging("fits")
        got = ctx.project(kind, vol)
        half = ctx.project(kind, vol, dtype=torch.bfloat16)
        ctx.set_tuning(rs_layout="plain")
        ref = ctx.project(kind, vol)
        torch.cuda.synchronize()
        assert ctx.errors() == 0
    assert float(ref.abs().max()) > 0 and torch.equal(got, ref)
    assert torch.equal(half, ref.to(torch.bfloat16))


@pytest.mark.parametrize("storage", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("spec", [(128, 128, 128, 128, 128, 45, 2.0), (131, 127, 130, 150, 141, 33, 1.7)],
                         ids=lambda s: "x".join(map(str, s)))
def test_half_staged_projection_equals_cells(tomo, spec, storage):
    """16-bit volumes from 128^3 on: some blocks stage slice pairs, the others gather them from
    the texture; bit-identical to the cell layout, from 16-bit volumes and, in the solver, from
    an FP32 iterate converted on the way (one iteration)."""
    cfg = _cfg(tomo, *spec)
    vol = torch.from_numpy(np.random.default_rng(8).random(cfg.volume_shape, dtype=np.float32)).cuda()
    real = torch.rand(cfg.sinogram_shape, device="cuda")
    par = tomo.GradientParams(gradient_iteration_nb=1, optimal_step_iteration_nb=2, real_f32=True,
                              storage="bf16" if storage == torch.bfloat16 else "f16")
    out = {}
    for lay in ("tex", "cell8"):
        with tomo.Context(cfg) as ctx:
            ctx.set_staging("fits")
            ctx.set_tuning(rs_layout=lay)
            assert ctx.rs_staged(storage) == (lay == "tex")
            out[lay] = [ctx.project(k, vol.to(storage), dtype=torch.float32) for k in ("RS", "RS_UM")]
            f = vol.clone()
            tomo.Solver(ctx, par).iterate(f, real)
            out[lay].append(f)  # the step's norm is summed per block: FP64 sums in another order
            torch.cuda.synchronize()
            assert ctx.errors() == 0
    for a, b in zip(out["tex"][:2], out["cell8"][:2]):
        assert float(b.abs().max()) > 0 and torch.equal(a, b)
    a, b = out["tex"][2], out["cell8"][2]
    assert float(torch.linalg.vector_norm((a - b).double()) / torch.linalg.vector_norm(b.double())) <= 1e-6


@pytest.mark.parametrize("tile", [(8, 16), (16, 64), (32, 128)])
def test_staged_projection_launch_shapes(tomo, tile):
    """Any block shape: the windows follow the tile."""
    cfg = _cfg(tomo, 70, 70, 50, 150, 61, 8, 1.0)
    vol = torch.rand(cfg.volume_shape, device="cuda")
    with tomo.Context(cfg) as ctx:
        ctx.set_staging("fits")
        ctx.set_tuning(rs_warp_u=tile[0], rs_tile_u=tile[1])
        got = ctx.project("RS", vol)
        ctx.set_tuning(rs_layout="plain")
        assert torch.equal(got, ctx.project("RS", vol))


# 4, 8 and 16 slices per thread (64^3, 128^3, 160^3), partial tiles and chunks, detector
# widths 0..3 modulo 4, a steep cone (windows beyond the box), a detector smaller than the
# volume's shadow
VI = [(64, 64, 64, 64, 64, 9, 2.0), (128, 128, 128, 130, 126, 5, 2.0), (160, 157, 161, 163, 141, 5, 2.0),
      (33, 41, 18, 47, 29, 7, 1.7), (96, 96, 200, 129, 240, 6, 3.0, 2.5, 80.0), (130, 130, 90, 61, 40, 6, 2.0)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("spec", VI, ids=lambda s: "x".join(map(str, s)))
def test_staged_backprojection_equals_padded(tomo, spec, dtype):
    """VI, its UM variant and FDK: bit-identical to the padded copy's kernel (32 slices per thread)."""
    cfg = _cfg(tomo, *spec)
    sino = torch.from_numpy(np.random.default_rng(5).random(cfg.sinogram_shape, dtype=np.float32)).cuda().to(dtype)
    with tomo.Context(cfg) as ctx:
        got = {k: ctx.backproject(k, sino, dtype=torch.float32) for k in ("VI", "VI_UM", "FDK")}
        ctx.set_tuning(vi_zc=2)
        for k, v in got.items():
            ref = ctx.backproject(k, sino, dtype=torch.float32)
            assert float(ref.abs().max()) > 0 and torch.equal(v, ref), k
        torch.cuda.synchronize()
        assert ctx.errors() == 0


def test_staged_copies_remade_at_the_same_address(tomo):
    """Copies of another type or size, made where earlier ones were freed: each projection is read
    through its own tensor maps (the type of one context's volume alternates; contexts of other
    sizes follow one another)."""
    for n, views in ((128, 45), (131, 45), (128, 44)):
        cfg = _cfg(tomo, n, n, n, n, n, views, 2.0)
        vol = torch.rand(cfg.volume_shape, device="cuda")
        with tomo.Context(cfg) as ctx, tomo.Context(cfg) as plain:
            ctx.set_staging("fits")
            plain.set_tuning(rs_layout="cell8")
            for dt in (torch.float32, torch.bfloat16, torch.float32, torch.float16, torch.bfloat16):
                v = vol.to(dt)
                assert torch.equal(ctx.project("RS", v, dtype=torch.float32), plain.project("RS", v, dtype=torch.float32)), (n, dt)


@pytest.mark.parametrize("dtype,n,views", [(torch.float32, 128, 8), (torch.bfloat16, 128, 45)])
def test_closed_contexts_give_their_copies_back(tomo, dtype, n, views):
    """A closed context leaves no device memory behind: its two volume copies are 16 MiB (FP32)
    at 128^3, so a leak of them shows after the second of six contexts."""
    cfg = _cfg(tomo, n, n, n, n, n, views, 2.0)
    vol = torch.rand(cfg.volume_shape, device="cuda").to(dtype)
    out = torch.empty(cfg.sinogram_shape, device="cuda", dtype=dtype)
    free = []
    for _ in range(6):
        with tomo.Context(cfg) as ctx:
            ctx.set_staging("fits")
            ctx.project("RS", vol, out=out)
            torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < 8 << 20, free


@pytest.mark.parametrize("dtype,n,views", [(torch.float32, 16, 4), (torch.bfloat16, 128, 40)])
def test_staged_projection_bounded_wait_reports_timeout(tomo, dtype, n, views):
    """With the test stall the producer issues no copy and the consumers' waits run out after
    their one-second bound: the call returns, ERR_TIMEOUT (bit 1) is in the context's error word,
    and the next call on the context is exact. A detector of one tile keeps it to a few blocks a
    view (16-bit volumes: the ones that do not gather)."""
    from tomogpi_b200 import _lib as L

    cfg = _cfg(tomo, n, n, n, 128 if n == 128 else 16, 128 if n == 128 else 8, views, 2.0)
    vol = torch.rand(cfg.volume_shape, device="cuda").to(dtype)
    with tomo.Context(cfg, views=(0, 1) if n == 16 else None) as ctx:
        ctx.set_staging("fits")
        ref = ctx.project("RS", vol)
        torch.cuda.synchronize()
        assert ctx.errors(clear=True) == 0
        L.call("tomo_context_test_stall", ctx.handle, 1)
        ctx.project("RS", vol)
        torch.cuda.synchronize()
        assert ctx.errors(clear=True) & 2
        L.call("tomo_context_test_stall", ctx.handle, 0)
        assert torch.equal(ctx.project("RS", vol), ref)
        assert ctx.errors() == 0


def test_copies_of_many_contexts_threads_and_streams(tomo):
    """The copies' memory outlives a context in its device's pool: contexts of several sizes, made
    and closed by four threads on streams of their own, each see their own copies."""
    import concurrent.futures as cf

    cfgs = [_cfg(tomo, n, n, n, n, n, 12, 2.0) for n in (40, 64, 100, 128)]
    vols = [torch.rand(c.volume_shape, device="cuda") for c in cfgs]
    refs = []
    for c, v in zip(cfgs, vols):
        with tomo.Context(c) as ctx:
            ctx.set_tuning(rs_layout="plain")
            refs.append(ctx.project("RS", v))
    torch.cuda.synchronize()

    def work(k):
        st, good = torch.cuda.Stream(), 0
        with torch.cuda.stream(st):
            for i in range(12):
                j = (k + i) % len(cfgs)
                with tomo.Context(cfgs[j]) as ctx:
                    ctx.set_staging("fits")
                    out = ctx.project("RS", vols[j])
                    st.synchronize()
                    good += int(torch.equal(out, refs[j]))
        return good

    with cf.ThreadPoolExecutor(4) as ex:
        assert list(ex.map(work, range(4))) == [12] * 4


@pytest.mark.parametrize("kind", ["VI", "VI_UM", "FDK"])
@pytest.mark.parametrize("offset", [0, 4, 1000])
def test_backprojection_over_its_sinogram(tomo, kind, offset):
    """The volume may lie over the sinogram that it comes from: the same values. 1000 blocks, so the
    later ones read what the first have written unless there is a copy."""
    n = 160
    cfg = _cfg(tomo, n, n, n, n, n, n, 2.0)
    buf = torch.empty(n ** 3 + offset, device="cuda")
    sino, vol = buf[:n ** 3].view(n, n, n), buf[offset:].view(n, n, n)
    src = torch.rand(n, n, n, device="cuda")
    with tomo.Context(cfg) as ctx:
        ref = ctx.backproject(kind, src)
        sino.copy_(src)
        assert torch.equal(ctx.backproject(kind, sino, out=vol), ref)


# (nx, ny, nz, nu, nv, views, pitch, mag[, fod]), FP32 staged?, 16-bit staged?
RULE = [((256, 256, 256, 256, 256, 64, 1.6), True, True), ((64, 64, 64, 64, 64, 60, 2.0), True, False),
        ((128, 128, 128, 256, 256, 60, 1.0), True, True), ((20, 20, 20, 20, 20, 60, 2.0), False, False),
        ((33, 33, 500, 33, 500, 30, 2.0), False, False), ((160, 160, 160, 123, 123, 40, 2.6, 2.0, 120.0), False, False),
        ((160, 160, 160, 133, 133, 60, 2.4), True, False), ((64, 64, 64, 20, 20, 9, 8.0), False, False)]


@pytest.mark.parametrize("spec,f32,half", RULE, ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else str(s))
def test_staged_where_it_is_faster(tomo, spec, f32, half):
    """The rule takes what the measurements behind it say, for both types, whatever was projected
    before; and the values do not depend on it (bit-identical to the padded layout)."""
    cfg = _cfg(tomo, *spec)
    vol = torch.rand(cfg.volume_shape, device="cuda")
    with tomo.Context(cfg) as ctx, tomo.Context(cfg) as plain:
        plain.set_tuning(rs_layout="plain")
        for dt, want in ((torch.float32, f32), (torch.bfloat16, half), (torch.float16, half), (torch.float32, f32)):
            assert ctx.rs_staged(dt) == want
            v = vol.to(dt)
            assert torch.equal(ctx.project("RS", v, dtype=torch.float32), plain.project("RS", v, dtype=torch.float32))
        ctx.set_tuning(rs_warp_u=32, rs_tile_u=128)
        ctx.set_tuning(rs_warp_u=8, rs_tile_u=32)
        assert ctx.rs_staged(torch.float32) == f32
