"""2D images through the strip kernels (several iterations per launch, tiles
held in registers) against the kernels that run one iteration per launch:
sizes at the edges of tiles and of strips, odd rows, images of one pixel
column or row, every choice of rows per thread, and the stopping rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (ny, nx): single pixels and rows, one tile, its edges, several tiles
SHAPES = [(1, 1), (1, 70), (70, 1), (2, 2), (3, 5), (33, 64), (64, 65), (97, 130), (131, 127), (200, 318)]
PLANS = ["2,1", "2,5", "3,7", "4,5", "4,16", "6,13"]


def _calls():
    from ccpi.filters import regularisersCuPy as R

    calls = {"rof": lambda f, it, tol, info: R.ROF_TV(f, 0.02, it, 0.001, tolerance_param=tol, infovector=info),
             "d4": lambda f, it, tol, info: R.Diff4th(f, 0.8, 0.02, it, 1e-4, tol, infovector=info),
             "llt": lambda f, it, tol, info: R.LLT_ROF(f, 0.02, 0.01, it, 1e-3, tol, infovector=info)}
    calls["tgv"] = lambda f, it, tol, info: R.TGV(f, 0.05, 1.0, 2.0, it, 12.0, tol, infovector=info)
    for a in (0, 1):  # isotropic; anisotropic and non-negative
        calls[f"fgp{a}"] = lambda f, it, tol, info, a=a: R.FGP_TV(f, 0.05, it, tol, a, a, infovector=info)
        calls[f"dtv{a}"] = lambda f, it, tol, info, a=a: R.FGP_dTV(f, f.flip(0).contiguous(), 0.05, it, tol, 0.2, a, a,
                                                                   infovector=info)
        calls[f"pd{a}"] = lambda f, it, tol, info, a=a: R.PD_TV(f, 0.05, it, tol, a, a, 8.0, infovector=info)
        calls[f"sb{a}"] = lambda f, it, tol, info, a=a: R.SB_TV(f, 0.05, it, tol, a, infovector=info)
    for p in range(6):  # 0: linear diffusion
        calls[f"ndf{p}"] = lambda f, it, tol, info, p=p: R.NDF(f, 0.02, 0.05 * (p > 0), it, 0.01, max(p, 1), tol,
                                                               infovector=info)
    return calls


def _image(shape, seed=3):
    import torch

    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0 : shape[0], 0 : shape[1]]
    img = ((x // 9 + y // 7) % 3) * 0.4 + rng.normal(0, 0.05, shape)
    return torch.from_numpy(img.astype(np.float32)).cuda()


def _run(monkeypatch, setting, op, f, it, tol=0.0):
    monkeypatch.setenv("CILREG_STRIP2D", setting)
    info = np.zeros(2, np.float32)
    out = _calls()[op](f, it, tol, info).cpu().numpy()
    monkeypatch.delenv("CILREG_STRIP2D")
    return out, info


OPS = ["rof", "d4", "llt", "fgp0", "fgp1", "dtv0", "dtv1", "pd0", "pd1", "sb0", "sb1", "tgv"] + [f"ndf{p}" for p in range(6)]


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", SHAPES)
def test_strips_equal_single_iterations(monkeypatch, op, shape):
    f = _image(shape)
    ref, _ = _run(monkeypatch, "0", op, f, 23)
    tol = 1e-5 * float(np.ptp(ref) or 1.0)
    for plan in PLANS:
        out, _ = _run(monkeypatch, plan, op, f, 23)
        if shape[1] % 2 == 0 and op in BIT_EQUAL:
            np.testing.assert_array_equal(out, ref, err_msg=plan)
        else:
            np.testing.assert_allclose(out, ref, rtol=0, atol=tol, err_msg=plan)


# the strip kernels that evaluate their one-iteration kernel's expressions one
# by one (even rows); SB's and TGV's leave fused operations to the compiler
BIT_EQUAL = set(OPS) - {"sb0", "sb1", "tgv"}


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", [(61, 90), (131, 127)])
def test_strips_stop_at_the_same_iteration(monkeypatch, op, shape):
    f = _image(shape)
    ref, want = _run(monkeypatch, "0", op, f, 203, 2e-3)
    for plan in ("2,5", "4,5", "1"):
        out, info = _run(monkeypatch, plan, op, f, 203, 2e-3)
        assert info[0] == want[0], plan
        np.testing.assert_allclose(info[1], want[1], rtol=1e-3)
        np.testing.assert_allclose(out, ref, rtol=0, atol=1e-5 * float(np.ptp(ref)))
    # the first check, and counts that end between checks
    for it in (1, 2, 5, 6, 9):
        ref, _ = _run(monkeypatch, "0", op, f, it, 1e-9)
        out, _ = _run(monkeypatch, "1", op, f, it, 1e-9)
        np.testing.assert_allclose(out, ref, rtol=0, atol=1e-5 * float(np.ptp(ref)))


@pytest.mark.parametrize("op", OPS)
def test_strips_take_arrays_off_8_byte_alignment(monkeypatch, op):
    import torch

    base = torch.zeros(1 + 77 * 130, device="cuda")
    f = base[1:].view(77, 130)
    f.copy_(_image((77, 130)))
    out, _ = _run(monkeypatch, "1", op, f, 17)
    ref, _ = _run(monkeypatch, "1", op, f.clone(), 17)
    np.testing.assert_array_equal(out, ref)


@pytest.mark.parametrize("op", ["fgp0", "fgp1", "dtv0", "dtv1", "rof"])
@pytest.mark.parametrize("shape", [(2, 3), (33, 63), (97, 131), (131, 127), (200, 319)])
def test_strips_of_odd_rows_keep_the_streaming_kernels_bits(monkeypatch, op, shape):
    f = _image(shape)
    for tol in (0.0, 1e-7):
        ref, _ = _run(monkeypatch, "0", op, f, 33, tol)
        for plan in ("1",) + tuple(PLANS):
            np.testing.assert_array_equal(_run(monkeypatch, plan, op, f, 33, tol)[0], ref, err_msg=plan)


@pytest.mark.parametrize("shapes", [[(37, 51), (128, 9), (201, 199), (1, 77)], [(36, 52), (128, 10), (200, 200)]],
                         ids=["odd rows", "even rows"])
@pytest.mark.parametrize("epsil", [0.0, 3e-4])
def test_fgp_batch_of_images_equals_single_calls(shapes, epsil):
    """As they run by default: strips in a single call, the batch's own kernel in the batch."""
    from ccpi.filters.batch import FGP_TV_batch
    from ccpi.filters.regularisers import FGP_TV

    rng = np.random.default_rng(5)
    vols = [rng.random(s).astype(np.float32) for s in shapes]
    lams = [0.03 + 0.01 * i for i in range(len(vols))]
    infos = np.zeros((len(vols), 2), np.float32)
    outs = FGP_TV_batch(vols, lams, 60, epsil, 0, 1, infovectors=infos)
    for v, o, lam, inf in zip(vols, outs, lams, infos):
        info = np.zeros(2, np.float32)
        np.testing.assert_array_equal(o, FGP_TV(v, lam, 60, epsil, 0, 1, device="gpu", infovector=info))
        assert int(inf[0]) == int(info[0])


@pytest.mark.parametrize("width", [64, 63])
@pytest.mark.parametrize("step", [1.0, 3.0])
def test_check_sums_lose_nothing_to_a_threads_other_rows(monkeypatch, width, step):
    """FGP's first iteration leaves U = f, so the check's relative change is known
    from f and the output's initial content.  Every fourth row's squares are 2^24
    times the others': one FP32 sum over a thread's four rows would lose those."""
    import ctypes

    import torch
    from ccpi.filters.utils import cilregcuda as C

    monkeypatch.setenv("CILREG_STRIP2D", "4,5")
    f = np.ones((64, width), np.float32)
    f[::4] = 4096.0
    prev = f - np.float32(step)
    d_f, d_u = torch.from_numpy(f).cuda(), torch.from_numpy(prev).cuda()
    info = (ctypes.c_float * 2)()
    assert C.cilreg_fgp_tv_dev(d_f.data_ptr(), d_u.data_ptr(), info, 0.05, 1, 1e-9, 0, 0, width, 64, 1,
                               torch.cuda.current_stream().cuda_stream) == 0
    np.testing.assert_array_equal(d_u.cpu().numpy(), f)
    a = ((f - prev).astype(np.float64) ** 2).sum()
    b = (f.astype(np.float64) ** 2).sum()
    assert np.float32(info[1]) == np.sqrt(np.float32(a)) / np.sqrt(np.float32(b))
