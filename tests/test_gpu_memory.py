"""What contexts and solvers do when a device allocation fails: the staged forms' buffers are
optional, so a call without room for them runs another form with the same result, and a call that
fails leaves an object that can be used again. The failures are injected on the host
(tomo_context_test_deny); nothing runs out of memory."""
import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tomo():
    import tomogpi_b200 as t

    return t


def _deny(ctx, skip, count):
    from tomogpi_b200 import _lib as L

    L.call("tomo_context_test_deny", ctx.handle, skip, count)


def _cfg(tomo, n=40, views=12):
    return tomo.ConfigCT.cone_beam(n, views)


def _context(tomo, cfg):
    """A context that stages its projections wherever the geometry allows it."""
    ctx = tomo.Context(cfg)
    ctx.set_staging("fits")
    return ctx


def _volume(cfg, seed=1):
    return torch.from_numpy(np.random.default_rng(seed).random(cfg.volume_shape, dtype=np.float32)).cuda()


def _sino(cfg, seed=2):
    return torch.from_numpy(np.random.default_rng(seed).random(cfg.sinogram_shape, dtype=np.float32)).cuda()


def test_projection_without_room_for_the_copies(tomo):
    """No room for the staged copies: the texture. Copies that give way to a later buffer: the
    texture from then on. Bit-identical either way."""
    cfg = _cfg(tomo)
    vol = _volume(cfg)
    with _context(tomo, cfg) as ctx:
        ref = ctx.project("RS", vol)
    with _context(tomo, cfg) as ctx:
        _deny(ctx, 1, 1)  # after the projector's input buffer
        assert torch.equal(ctx.project("RS", vol), ref)
        assert torch.equal(ctx.project("RS", vol), ref)
    with _context(tomo, cfg) as ctx:
        ctx.project("RS", vol)
        _deny(ctx, 0, 1)  # the host form's volume
        assert np.array_equal(ctx.project_host("RS", vol.cpu().numpy()), ref.cpu().numpy())
        assert torch.equal(ctx.project("RS", vol), ref)
    with _context(tomo, cfg) as ctx:
        _deny(ctx, 1, 2)  # neither the copies nor the texture
        with pytest.raises(RuntimeError, match="NO_MEMORY"):
            ctx.project("RS", vol)
        assert torch.equal(ctx.project("RS", vol), ref)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_backprojection_without_room_for_the_rows(tomo, dtype):
    """No room for the FP32 rows: the padded copy, bit-identical; nor for that one: an error, and
    the next call runs."""
    cfg = _cfg(tomo).replace(u_detector_pixel_nb=42)
    s = _sino(cfg).to(dtype)
    with _context(tomo, cfg) as ctx:
        ref = ctx.backproject("VI", s, dtype=torch.float32)
    with _context(tomo, cfg) as ctx:
        _deny(ctx, 0, 2)
        with pytest.raises(RuntimeError, match="NO_MEMORY"):
            ctx.backproject("VI", s, dtype=torch.float32)
        _deny(ctx, 0, 1)
        assert torch.equal(ctx.backproject("VI", s, dtype=torch.float32), ref)
        assert torch.equal(ctx.backproject("VI", s, dtype=torch.float32), ref)


def _params(tomo, **kw):
    return tomo.GradientParams(gradient_iteration_nb=2, optimal_step_iteration_nb=3, regularization_parameter=0.01, **kw)


@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_solver_creation_with_one_failed_allocation(tomo, storage):
    """Whichever single allocation fails, creation reports it or the solver runs without it."""
    cfg = _cfg(tomo)
    s = _sino(cfg)
    par = _params(tomo, storage=storage, real_f32=True)
    with _context(tomo, cfg) as ctx:
        ref = tomo.Solver(ctx, par).iterate(_volume(cfg), s).cpu().numpy()
        made = 0
        for skip in range(14):
            _deny(ctx, skip, 1)
            try:
                sv = tomo.Solver(ctx, par)
            except RuntimeError as e:
                assert "NO_MEMORY" in str(e)
                continue
            _deny(ctx, 0, 0)
            made += 1
            assert rel_l2(sv.iterate(_volume(cfg), s).cpu().numpy(), ref) <= 1e-6, skip
            sv.close()
        assert made >= 2  # one without the failure at least


@pytest.mark.parametrize("fails", [1, 2, 3, 4])
@pytest.mark.parametrize("step", ["huber", "weights", "host"])
def test_solver_whose_copies_gave_way(tomo, step, fails):
    """A buffer that does not fit makes the solver's staged copies give way (1); the texture that
    takes their place may not fit either (2), nor at the next iterations (3, 4). Every failing
    call raises before it launches anything, and the solver then gives the same result."""
    cfg = _cfg(tomo)
    s = _sino(cfg)
    w = torch.rand(cfg.sinogram_shape, device="cuda") + 0.5

    def run(solver, deny):
        tries = 0

        def insist(f):
            nonlocal tries
            for _ in range(6):
                try:
                    return f()
                except RuntimeError as e:
                    assert "NO_MEMORY" in str(e)
                    tries += 1
            raise AssertionError("still no memory")

        if deny:
            _deny(solver.ctx, 0, deny)
        if step == "host":
            vol = _volume(cfg).cpu().numpy()
            insist(lambda: solver.iterate_host(vol, s.cpu().numpy()))
            return vol, tries
        f = (lambda: solver.set_regularizer("huber", 0.02)) if step == "huber" else (lambda: solver.set_weights(w))
        if deny >= 2:  # the failed call's buffer was not handed out; iterations go on without it
            with pytest.raises(RuntimeError, match="NO_MEMORY"):
                f()
            tries += 1
            insist(lambda: solver.iterate(_volume(cfg), s, first=1, count=0))
            solver.set_state(-0.0347711, 1)
        insist(f)
        vol = _volume(cfg)
        insist(lambda: solver.iterate(vol, s))
        return vol.cpu().numpy(), tries

    with _context(tomo, cfg) as ctx:
        ref, none = run(tomo.Solver(ctx, _params(tomo)), 0)
        got, tries = run(tomo.Solver(ctx, _params(tomo)), fails)
        _deny(ctx, 0, 0)
    assert none == 0 and (tries > 0) == (fails > 1)
    assert rel_l2(got, ref) <= 1e-6


def _captured(f):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f()
    return g


def test_captured_launches_keep_their_buffers(tomo):
    """The copies and rows that a captured projection or backprojection reads never give way, to a
    buffer or to a volume of another type: the replay is exact after either."""
    cfg = _cfg(tomo, n=128, views=45).replace(u_detector_pixel_nb=126)
    vol, s = _volume(cfg), _sino(cfg).to(torch.bfloat16)
    with _context(tomo, cfg) as ctx:
        fwd, back = ctx.project("RS", vol), ctx.backproject("VI", s, dtype=torch.float32)
        ref, bref = fwd.clone(), back.clone()
        g = _captured(lambda: (ctx.project("RS", vol, out=fwd), ctx.backproject("VI", s, out=back)))
        _deny(ctx, 0, 1)
        with pytest.raises(RuntimeError, match="NO_MEMORY"):
            ctx.project_host("RS", vol.cpu().numpy())
        half = ctx.project("RS", vol.to(torch.bfloat16), dtype=torch.float32)
        fwd.zero_(), back.zero_()
        g.replay()
        assert torch.equal(fwd, ref) and torch.equal(back, bref)
        ctx.set_tuning(rs_layout="cell8")
        assert torch.equal(half, ctx.project("RS", vol.to(torch.bfloat16), dtype=torch.float32))
        torch.cuda.synchronize()
        del g


def test_captured_iterations_keep_the_solvers_copies(tomo):
    """The same for the copies that a solver's captured iterations read."""
    cfg = _cfg(tomo)
    s = _sino(cfg)
    with _context(tomo, cfg) as ctx:
        sv = tomo.Solver(ctx, _params(tomo))
        vol = _volume(cfg)
        ref = sv.iterate(vol, s).clone()
        g = _captured(lambda: sv.iterate(vol, s))
        _deny(ctx, 0, 1)
        with pytest.raises(RuntimeError, match="NO_MEMORY"):
            sv.set_regularizer("huber", 0.02)
        sv.set_state(-0.0347711, 1)
        vol.copy_(_volume(cfg))
        g.replay()
        assert rel_l2(vol.cpu().numpy(), ref.cpu().numpy()) <= 1e-6
        torch.cuda.synchronize()
        del g


def test_copies_give_way_to_a_new_solver(tomo):
    """A solver that finds no room takes that of the context's copies and rows."""
    cfg = _cfg(tomo).replace(u_detector_pixel_nb=42)
    vol, s = _volume(cfg), _sino(cfg)
    with _context(tomo, cfg) as ctx:
        ref = tomo.Solver(ctx, _params(tomo)).iterate(vol.clone(), s)
    with _context(tomo, cfg) as ctx:
        fwd, back = ctx.project("RS", vol), ctx.backproject("VI", s)
        _deny(ctx, 1, 1)
        assert rel_l2(tomo.Solver(ctx, _params(tomo)).iterate(vol.clone(), s).cpu().numpy(), ref.cpu().numpy()) <= 1e-6
        assert torch.equal(ctx.project("RS", vol), fwd) and torch.equal(ctx.backproject("VI", s), back)


def test_capture_with_a_sinogram_that_needs_rows(tomo):
    """Whether a backprojection copies its FP32 rows depends on the sinogram's address: a call that
    ran on an aligned one can be captured on another."""
    cfg = _cfg(tomo)
    s = _sino(cfg)
    odd = torch.empty(s.numel() + 1, device="cuda")[1:].view(s.shape).copy_(s)
    with _context(tomo, cfg) as ctx:
        back = ctx.backproject("VI", s)
        ref = back.clone()
        back.zero_()
        g = _captured(lambda: ctx.backproject("VI", odd, out=back))
        g.replay()
        assert torch.equal(back, ref)
        torch.cuda.synchronize()
        del g


@pytest.mark.parametrize("what", ["project", "backproject", "iterate"])
def test_host_forms_report_a_wait_that_gave_up(tomo, what):
    """A bounded wait that runs out (the test stall: no copies are issued) fails a call on host
    buffers with TOMO_ERR_TIMEOUT; the next call is exact. One view of a tiny volume."""
    from tomogpi_b200 import _lib as L

    cfg = tomo.ConfigCT.cone_beam(16, 4)
    vol = np.random.default_rng(3).random(cfg.volume_shape, dtype=np.float32)
    with tomo.Context(cfg, views=(0, 1)) as ctx:
        ctx.set_staging("fits")
        s = np.random.default_rng(4).random(ctx.sinogram_shape, dtype=np.float32)
        sv = tomo.Solver(ctx, _params(tomo))
        call = {"project": lambda: ctx.project_host("RS", vol), "backproject": lambda: ctx.backproject_host("VI", s),
                "iterate": lambda: sv.iterate_host(vol.copy(), s, first=1, count=1)}[what]
        ref = call()
        L.call("tomo_context_test_stall", ctx.handle, 1)
        with pytest.raises(L.TomoError, match="TIMEOUT"):
            call()
        L.call("tomo_context_test_stall", ctx.handle, 0)
        sv.set_state(-0.0347711, 1)
        assert np.array_equal(call(), ref) and ctx.errors() == 0
