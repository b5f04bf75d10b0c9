"""The interval steppers at the edges of their tiles: strips of one row quad and of a remainder, chunks
narrower than a block, idle lanes, one and many strips, launches that straddle a coarse interval
(sub > 4), against the per-fine-step stepper. Both are FP32 evaluations of one scheme: relative L2 below
2e-5 (each is within 1e-5 of the FP64 oracle at these lengths, tests/test_gpu_parity.py)."""
import numpy as np
import pytest

from cases import interior_mask, make_case, rel_l2

pytestmark = pytest.mark.gpu

# nzi, nxi, shots: below one warp of row quads, exactly one (128 rows) and one row more, two strips, odd sizes
SIZES = [(11, 23, 1), (33, 40, 3), (128, 37, 2), (129, 61, 1), (301, 45, 2), (67, 530, 1), (530, 30, 1)]


def _pair(nzi, nxi, sub, fs, shots, chunk=0, **kw):
    import orc
    from acoustic_isotropic_operators_b200.batch import Context
    c = make_case(seed=nzi + sub, nzi=nzi, nxi=nxi, nts=14, sub=sub, minPad=6, nshots=shots, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    mk = lambda **a: Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], free_surface=fs,  # noqa: E731
                             **kw, **a)
    return c, mk(chunk_columns=chunk), mk(stepper="fine")


def _shots(c, data=None):
    from acoustic_isotropic_operators_b200.batch import Shot
    return [Shot(c.src_pos[i], c.rec_pos[i], c.sig[i], None if data is None else data[i]) for i in range(len(c.src_pos))]


@pytest.mark.parametrize("fs", [0, 1])
@pytest.mark.parametrize("sub", [4, 5, 7, 8])
@pytest.mark.parametrize("nzi,nxi,shots", SIZES)
def test_against_fine_steps(nzi, nxi, shots, sub, fs):
    """Timed plans, and (chunk 17) marching strips of at most 128 rows."""
    for chunk in (0, 17):
        c, blocked, fine = _pair(nzi, nxi, sub, fs, shots, chunk)
        data = [c.rng.standard_normal((len(r), c.scheme.nts)).astype(np.float32) for r in c.rec_pos]
        model = (c.rng.standard_normal((c.nx, c.nz)) * interior_mask(c.nx, c.nz)).astype(np.float32)
        out = []
        for ctx in (blocked, fine):
            out.append([np.concatenate([x.ravel() for x in ctx.nonlinear_forward(_shots(c))]),
                        np.concatenate([x.ravel() for x in ctx.nonlinear_adjoint(_shots(c, data))]),
                        np.concatenate([x.ravel() for x in ctx.born_forward(model, _shots(c))]),
                        ctx.born_adjoint(_shots(c, data)).ravel().copy()])
            ctx.close()
        for name, a, b in zip(("nl fwd", "nl adj", "born fwd", "born adj"), *out):
            assert np.linalg.norm(b) > 0
            assert rel_l2(a, b) < 2e-5, (name, chunk)


@pytest.mark.parametrize("nzi,nxi,shots", SIZES)
def test_dense_source_passes(nzi, nxi, shots):
    """Tomo (dense sources, stored samples), timed plans."""
    c, blocked, fine = _pair(nzi, nxi, 4, 0, shots, nExt=3)
    ext = (c.rng.standard_normal((3, c.nx, c.nz)) * interior_mask(c.nx, c.nz)).astype(np.float32)
    data = [c.rng.standard_normal((len(r), c.scheme.nts)).astype(np.float32) for r in c.rec_pos]
    out = []
    for ctx in (blocked, fine):
        out.append([np.concatenate([x.ravel() for x in ctx.tomo_forward(ext[1], ext, _shots(c))]),
                    ctx.tomo_adjoint(ext, _shots(c, data)).ravel().copy()])
        ctx.close()
    for a, b in zip(*out):
        assert np.linalg.norm(b) > 0
        assert rel_l2(a, b) < 1e-4  # (second differences of FP32 fields)


@pytest.mark.parametrize("sub", [4, 6])
def test_devices_everywhere(sub):
    """A receiver on every third grid point and two devices on one point: more entries per CTA than the
    preferred tiles hold, recordings and injections in every warp."""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    c = make_case(seed=9, nzi=140, nxi=90, nts=10, sub=sub, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    pos = np.array([ix * s.nz + iz for ix in range(5, s.nx - 5) for iz in range(5, s.nz - 5)][::3], np.int32)
    pos = np.concatenate([pos, pos[:1]])
    data = (c.rng.standard_normal((len(pos), s.nts)) * 1e-2).astype(np.float32)
    out = []
    for stepper in ("auto", "fine"):
        ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], stepper=stepper)
        out.append([ctx.nonlinear_forward([Shot(c.src_pos[0], pos, c.sig[0])])[0].copy(),
                    ctx.nonlinear_adjoint([Shot(c.src_pos[0], pos, None, data)])[0].copy(),
                    ctx.born_adjoint([Shot(c.src_pos[0], pos, c.sig[0], data)]).copy()])
        ctx.close()
    np.testing.assert_array_equal(out[0][0][0], out[0][0][-1])
    for a, b in zip(*out):
        assert rel_l2(a, b) < 2e-5


@pytest.mark.parametrize("chunk", [0, 200])
def test_plans_follow_the_devices(chunk):
    """A plan timed (or forced) for few devices gives way to smaller tiles when a later call's do not fit."""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    c = make_case(seed=4, nzi=210, nxi=200, nts=8, sub=4, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    block = np.array([ix * s.nz + iz for ix in range(60, 160) for iz in range(60, 130)], np.int32)
    # the source inside the block: 40 points away what arrives in 28 steps is subnormal (10 stencil hops of
    # about 1e-4 each), where FP32 results differ by their last bits, 1e-3 of the value
    src = block[3535:3536]
    sig = c.sig[0][:1]
    out = []
    for a in (dict(chunk_columns=chunk), dict(stepper="fine")):
        ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], **a)
        res = []
        for pos in (block[3600:3603], block, block[3600:3603]):
            data = (np.random.default_rng(2).standard_normal((len(pos), s.nts)) * 1e-2).astype(np.float32)
            res += [ctx.nonlinear_forward([Shot(src, pos, sig)])[0].copy(),
                    ctx.nonlinear_adjoint([Shot(src, pos, None, data)])[0].copy(),
                    ctx.born_adjoint([Shot(src, pos, sig, data)]).copy()]
        out.append(res)
        ctx.close()
    for a, b in zip(*out):
        assert rel_l2(a, b) < 2e-5


def test_small_budgets_take_fine_steps():
    """The nonlinear adjoint and sub > 4 fall back to the per-fine-step stepper (same bits) where a wave of
    the interval steppers would not fit the budget; at sub = 4 the forward is refused, as it always was."""
    from acoustic_isotropic_operators_b200._capi import AioError
    for sub in (4, 6):
        c, blocked, fine = _pair(61, 50, sub, 0, 1)
        blocked.set_budget(40 << 20)  # (below the 64 MiB a blocked wave sets aside)
        data = [c.rng.standard_normal((len(r), c.scheme.nts)).astype(np.float32) for r in c.rec_pos]
        np.testing.assert_array_equal(blocked.nonlinear_adjoint(_shots(c, data))[0], fine.nonlinear_adjoint(_shots(c, data))[0])
        if sub == 4:
            with pytest.raises(AioError):
                blocked.nonlinear_forward(_shots(c))
        else:
            np.testing.assert_array_equal(blocked.nonlinear_forward(_shots(c))[0], fine.nonlinear_forward(_shots(c))[0])
            np.testing.assert_array_equal(blocked.born_adjoint(_shots(c, data)), fine.born_adjoint(_shots(c, data)))
        blocked.close()
        fine.close()


@pytest.mark.parametrize("extension", ["time", "offset"])
@pytest.mark.parametrize("nExt,nzi,nxi,nts", [(1, 33, 23, 5), (3, 40, 24, 34), (9, 129, 25, 33), (17, 35, 64, 41), (19, 37, 67, 66)])
def test_extended_blocks(nExt, nzi, nxi, nts, extension):
    """Blocks of samples at the edges of their groups: lags around 8 and 16, samples around 32, columns around
    8, offsets wider than the grid allows."""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context
    c = make_case(seed=nExt, nzi=nzi, nxi=nxi, nts=nts, sub=4, minPad=6, nshots=2, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    ext = (c.rng.standard_normal((nExt, c.nx, c.nz)) * interior_mask(c.nx, c.nz)).astype(np.float32)
    data = [c.rng.standard_normal((len(r), s.nts)).astype(np.float32) for r in c.rec_pos]
    out = []
    for a in ({}, dict(stepper="fine")):
        ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], nExt=nExt, extension=extension, **a)
        out.append([np.concatenate([x.ravel() for x in ctx.born_ext_forward(ext, _shots(c))]),
                    ctx.born_ext_adjoint(_shots(c, data)).ravel().copy()])
        ctx.close()
    for a, b in zip(*out):
        assert np.linalg.norm(b) > 0
        assert rel_l2(a, b) < 3e-5


def test_staged_models():
    """Models of 16 MiB and more in pageable memory (copied directly until a context has moved 80 MiB of them, then
    packed through pinned buffers: four of them a round here, 18 MiB each) and in pinned memory (copied directly): the
    same bits, zeros outside the interior, the caller's array added to."""
    import orc
    import torch
    from acoustic_isotropic_operators_b200.batch import Context
    c = make_case(seed=8, nzi=301, nxi=403, nts=6, sub=4, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], nExt=37)
    mask = interior_mask(c.nx, c.nz)
    ext = (c.rng.standard_normal((37, c.nx, c.nz)) * mask).astype(np.float32)
    start = c.rng.standard_normal(ext.shape).astype(np.float32)
    data = [c.rng.standard_normal((len(r), s.nts)).astype(np.float32) for r in c.rec_pos]
    out = []
    for pin in (False, False, False, True):
        own = (lambda a: torch.from_numpy(a).pin_memory().numpy()) if pin else np.copy
        res = [np.concatenate([x.ravel() for x in ctx.born_ext_forward(own(ext), _shots(c))])]
        for add in (False, True):
            m = own(start)
            ctx.born_ext_adjoint(_shots(c, data), model=m, add=add)
            res.append(m.copy())
        out.append(res)
    ctx.close()
    for res in out[1:]:
        for a, b in zip(out[0], res):
            np.testing.assert_array_equal(a, b)
    edge = np.broadcast_to(mask == 0, ext.shape)
    assert not out[0][1][edge].any() and np.linalg.norm(out[0][1]) > 0
    np.testing.assert_array_equal(out[0][2][edge], start[edge])


@pytest.mark.parametrize("sub", [4, 6])
@pytest.mark.parametrize("chunk", [0, 17])
def test_devices_of_one_point_add_up_in_list_order(chunk, sub):
    """Devices of one point inject their sum in list order, as the per-fine-step stepper does. Here each sum
    is of B, v and -B in turn with |v| < |B| 2^-25: exactly zero in that order (B + v = B) and v at least
    in another one."""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    c = make_case(seed=12, nzi=90, nxi=70, nts=10, sub=sub, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    # points around chunk edges and strips, their devices interleaved in the list
    points = np.array([(5 + ix) * s.nz + 5 + iz for ix in (2, 16, 17, 18, 40, 69) for iz in (0, 3, 45, 89)], np.int32)
    pos = np.tile(points, 12)
    rng = np.random.default_rng(5)
    def traces(n):  # noqa: E306
        v = rng.standard_normal((4, len(points), n)).astype(np.float32)
        return np.concatenate([x for t in v for x in (t * np.float32(2.0 ** 27), t, -t * np.float32(2.0 ** 27))])
    far = np.array([30 * s.nz + 40], np.int32)
    out = {}
    for name, a in (("auto", dict(chunk_columns=chunk)), ("fine", dict(stepper="fine"))):
        ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], **a)
        rng = np.random.default_rng(5)
        out[name] = [ctx.nonlinear_forward([Shot(pos, points, traces(s.ntw))])[0],
                     ctx.nonlinear_adjoint([Shot(far, pos, None, traces(s.nts))])[0]]
        ctx.close()
    for x in out["fine"] + out["auto"]:
        assert not x.any()


def test_adjoint_without_velocity():
    """Where v^2 is zero at a source the nonlinear adjoint keeps the per-fine-step stepper (same bits), also
    when the velocity was taken away after the context was made."""
    from acoustic_isotropic_operators_b200 import _capi as A
    from acoustic_isotropic_operators_b200.batch import Shot
    c, auto, fine = _pair(40, 50, 4, 0, 2)
    data = [c.rng.standard_normal((len(r), c.scheme.nts)).astype(np.float32) for r in c.rec_pos]
    shots = lambda: [Shot(s, np.concatenate([r, s]), None, np.concatenate([d, d[:len(s)]]))  # noqa: E731
                     for s, r, d in zip(c.src_pos, c.rec_pos, data)]
    moving = auto.nonlinear_adjoint(shots())
    for ctx in (auto, fine):
        A.check(A.lib().aio_context_set_velocity(ctx._h, None, None))
    for a, b in zip(auto.nonlinear_adjoint(shots()), fine.nonlinear_adjoint(shots())):
        assert np.isfinite(a).all() and b.any()
        np.testing.assert_array_equal(a, b)
    auto.close()
    fine.close()
    assert all(x.any() for x in moving)


@pytest.mark.parametrize("sub", [4, 6])
def test_counts_without_positions(sub):
    """A device count without positions is no device, on either stepper."""
    from acoustic_isotropic_operators_b200 import _capi as A
    c, auto, fine = _pair(40, 50, sub, 0, 1)
    s = c.scheme
    pos, data = c.rec_pos[0], c.rng.standard_normal((len(c.rec_pos[0]), s.nts)).astype(np.float32)
    sig, out = np.ones((2, s.ntw), np.float32), []
    for ctx in (auto, fine):
        res = np.full((len(pos), s.nts), 7.0, np.float32), np.full((2, s.ntw), 7.0, np.float32)
        A.check(A.lib().aio_nonlinear_forward(ctx._h, 1, (A.AioShot * 1)(A.AioShot(
            None, 2, A.iptr(pos), len(pos), A.fptr(sig), A.fptr(res[0]), None, None)), A.AIO_MEM_HOST))
        A.check(A.lib().aio_nonlinear_adjoint(ctx._h, 1, (A.AioShot * 1)(A.AioShot(
            None, 2, A.iptr(pos), len(pos), None, A.fptr(data), None, A.fptr(res[1]))), A.AIO_MEM_HOST))
        out += res
        ctx.close()
    assert not any(x.any() for x in out)


def test_more_shots_than_a_grid_holds():
    """More shots than one launch can index (65535) run in waves."""
    from acoustic_isotropic_operators_b200.batch import Shot
    c, auto, fine = _pair(11, 13, 4, 0, 3)
    data = [c.rng.standard_normal((len(r), c.scheme.nts)).astype(np.float32) for r in c.rec_pos]
    want = fine.nonlinear_adjoint(_shots(c, data))
    n = 65538
    got = auto.nonlinear_adjoint([Shot(c.src_pos[i % 3], c.rec_pos[i % 3], None, data[i % 3]) for i in range(n)])
    for i in range(3):
        same = np.stack(got[i::3])
        np.testing.assert_array_equal(same, np.broadcast_to(same[0], same.shape))
        assert rel_l2(same[0], want[i]) < 2e-5 and want[i].any()
    auto.close()
    fine.close()


def test_both_steppers_share_the_budget():
    """At sub != 4 the Born operators and the extended ones keep their fields on different steppers: a context
    that runs both in turn stays within its budget."""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    c = make_case(seed=3, nzi=61, nxi=50, nts=300, sub=6, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], nExt=3)
    budget = 200 << 20  # (about 30 of the 40 shots, of 3.8 MB of coarse source field each)
    ctx.set_budget(budget)
    data = (c.rng.standard_normal((len(c.rec_pos[0]), s.nts)) * 1e-2).astype(np.float32)
    shots = [Shot(c.src_pos[0], c.rec_pos[0], c.sig[0], data) for _ in range(40)]
    out = []
    for _ in range(2):
        out.append((ctx.born_adjoint(shots), ctx.born_ext_adjoint(shots)))
        assert ctx.device_bytes <= budget
    ctx.close()
    for a, b in zip(*out):
        assert a.any()
        np.testing.assert_array_equal(a, b)


def test_few_devices_after_many(monkeypatch, capfd):
    """A call of few devices is not left with the plan that a call of many had to take, in the same context
    or in another one of the process; neither is timed twice. (The grids are this test's own.)"""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    monkeypatch.setenv("AIO_AUTOTUNE_LOG", "1")
    c = make_case(seed=4, nzi=214, nxi=204, nts=8, sub=4, minPad=6, nshots=1, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    points = np.array([[ix * s.nz + iz for iz in range(5, s.nz - 5)] for ix in range(5, s.nx - 5)], np.int32)
    # held by every, by some and by none of the timed tiles
    few, some, many = points[70, 60:63], points[60:160, 60:130].ravel(), points.ravel()
    ctx = [Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"]) for _ in range(3)]

    def plan(i, pos):
        capfd.readouterr()
        data = np.zeros((len(pos), s.nts), np.float32)
        ctx[i].nonlinear_adjoint([Shot(c.src_pos[0], pos, None, data) for _ in range(6)])
        return ctx[i].blocked_plan(0), capfd.readouterr().err.count("aio autotune")

    first = plan(0, many), plan(0, some), plan(0, few)
    assert first[0][1] == 0 and 0 < first[1][1] < first[2][1]
    plans = [p for p, _ in first]
    for i, pos, want in ((0, some, plans[1:]), (0, few, plans[2:]), (0, many, plans[:1]),
                         (1, many, plans[:1]), (1, few, plans[2:]), (2, some, plans[1:]), (2, few, plans[2:])):
        got, timed = plan(i, pos)
        assert got in want and timed == 0
    for x in ctx:
        x.close()


# as SIZES, wide enough for several plans of every kind (a tile's chunks are a multiple of four columns, of 8 at least)
KIND_SIZES = [(21, 48, 1), (33, 40, 3), (128, 64, 2), (129, 61, 1), (301, 45, 2), (67, 530, 1), (530, 32, 1)]


@pytest.mark.parametrize("nzi,nxi,shots,fs,wavefield",
                         [(*s, fs, "fp32") for s in KIND_SIZES for fs in (0, 1)] +
                         [(*s, fs, w) for s in KIND_SIZES[2:5] for fs in (0, 1) for w in ("bf16", "fp16")])
def test_stepper_kernels_agree(nzi, nxi, shots, fs, wavefield, monkeypatch, capfd):
    """The marching, tile and sliding-block kernels give the same bits at sub = 4 in every operator, so that the
    timed choice between them changes no result. (The sliding blocks run the dense-source passes only.)"""
    import orc
    from acoustic_isotropic_operators_b200.batch import Context, Shot
    monkeypatch.setenv("AIO_AUTOTUNE_LOG", "1")
    c = make_case(seed=nzi + 7, nzi=nzi, nxi=nxi, nts=14, sub=4, minPad=6, nshots=shots, vmin=1500.0, vmax=1900.0)
    s = c.scheme
    k = orc.constants(s, c.vel, dtype=np.float32)
    ext = (c.rng.standard_normal((3, c.nx, c.nz)) * interior_mask(c.nx, c.nz)).astype(np.float32)
    data = [c.rng.standard_normal((len(r), s.nts)).astype(np.float32) for r in c.rec_pos]
    wemva = lambda: [Shot(c.src_pos[i], c.rec_pos[i], c.sig[i], None, data[i]) for i in range(shots)]  # noqa: E731
    out = {}
    for kind in ("march", "tile", "slide"):
        monkeypatch.setenv("AIO_PLANS", kind)
        capfd.readouterr()
        ctx = Context(s.nz, s.nx, s.nts, s.dts, s.sub, s.dz, s.dx, s.minPad, k["v2"], k["rs"], nExt=3, free_surface=fs,
                      wavefield=wavefield)
        flat = lambda x: np.concatenate([a.ravel() for a in x])  # noqa: E731
        out[kind] = {"nl fwd": flat(ctx.nonlinear_forward(_shots(c))), "nl adj": flat(ctx.nonlinear_adjoint(_shots(c, data))),
                     "born fwd": flat(ctx.born_forward(ext[1], _shots(c))), "born adj": ctx.born_adjoint(_shots(c, data)),
                     "ext fwd": flat(ctx.born_ext_forward(ext, _shots(c))), "ext adj": ctx.born_ext_adjoint(_shots(c, data)),
                     "tomo fwd": flat(ctx.tomo_forward(ext[1], ext, _shots(c))),
                     "tomo adj": ctx.tomo_adjoint(ext, _shots(c, data)),
                     "wemva fwd": ctx.wemva_forward(ext[1], wemva()), "wemva adj": ctx.wemva_adjoint(ext, wemva())}
        ctx.close()
        log = [x for x in capfd.readouterr().err.splitlines() if x.startswith("aio autotune")]
        # classes: light 0, heavy 1, receiver 2, nonlinear 3 and 4, dense 5
        own = [x.split("class ")[1][0] for x in log if (f"({kind})" in x if kind != "march" else "(" not in x)]
        assert set(own) == (set("15") if kind == "slide" else set("012345"))
    for kind in ("tile", "slide"):
        for op, want in out["march"].items():
            assert want.any(), op
            np.testing.assert_array_equal(out[kind][op], want, err_msg=f"{kind} {op}")
