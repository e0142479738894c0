"""Stream order at both ends of a call.  The input may come from a kernel that
has triggered its dependents (programmatic dependent launch) and still writes it
when the call's first kernel starts; and a call that has returned has nothing
left to write, so that its output may be read from any stream."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRODUCER = r"""
// triggers at once, waits a tenth of a millisecond (at most 10 ms), then copies
__global__ void k_late(const float* src, float* dst, long long n) {
    asm volatile("griddepcontrol.launch_dependents;");
    const long long t0 = clock64();
    for (int i = 0; i < 100000 && clock64() - t0 < 200000; i++) __nanosleep(100);
    for (long long i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}
extern "C" int late_copy(const float* src, float* dst, long long n, void* stream) {
    k_late<<<1, 1024, 0, (cudaStream_t)stream>>>(src, dst, n);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def late_copy(tmp_path_factory):
    d = tmp_path_factory.mktemp("producer")
    src, lib = d / "late.cu", d / "late.so"
    src.write_text(PRODUCER)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    assert os.path.exists(nvcc)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler", "-fPIC", "-o",
                    str(lib), str(src)], check=True)
    fn = ctypes.CDLL(str(lib)).late_copy
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]

    def run(src, dst):
        import torch

        assert fn(src.data_ptr(), dst.data_ptr(), src.numel(), torch.cuda.current_stream().cuda_stream) == 0

    return run


def _dev_calls():
    """Each regulariser's device-pointer entry point as call(f, out, iters, epsil, info, stream), 2D."""
    from ccpi.filters.utils import cilregcuda as C

    V, F, I = ctypes.c_void_p, ctypes.c_float, ctypes.c_int

    def call(name, f, out, info, stream, *rest):
        fn = getattr(C, name)
        args = [V(f.data_ptr()), V(out.data_ptr()), info.ctypes.data_as(ctypes.POINTER(F))] + list(rest)
        ny, nx = f.shape
        assert fn(*args, I(nx), I(ny), I(1), V(stream)) == 0

    def dtv(f, out, it, eps, info, s):
        ny, nx = f.shape
        assert C.cilreg_dtv_fgp_dev(V(f.data_ptr()), V(dtv.ref.data_ptr()), V(out.data_ptr()),
                                    info.ctypes.data_as(ctypes.POINTER(F)), F(0.05), I(it), F(eps), F(0.2), I(0), I(0),
                                    I(nx), I(ny), I(1), V(s)) == 0

    return {
        "rof": lambda f, o, it, eps, i, s: call("cilreg_rof_tv_dev", f, o, i, s, None, F(0.02), I(it), F(0.001), F(eps)),
        "fgp": lambda f, o, it, eps, i, s: call("cilreg_fgp_tv_dev", f, o, i, s, F(0.05), I(it), F(eps), I(0), I(0)),
        "pd": lambda f, o, it, eps, i, s: call("cilreg_pd_tv_dev", f, o, i, s, F(0.05), I(it), F(eps), F(8.0), I(0), I(0)),
        "sb": lambda f, o, it, eps, i, s: call("cilreg_sb_tv_dev", f, o, i, s, F(0.05), I(it), F(eps), I(0)),
        "tgv": lambda f, o, it, eps, i, s: call("cilreg_tgv_dev", f, o, i, s, F(0.05), F(1.0), F(2.0), I(it), F(12.0), F(eps)),
        "ndf": lambda f, o, it, eps, i, s: call("cilreg_ndf_dev", f, o, i, s, F(0.02), F(0.05), I(it), F(0.01), I(1), F(eps)),
        "d4": lambda f, o, it, eps, i, s: call("cilreg_diff4th_dev", f, o, i, s, F(0.8), F(0.02), I(it), F(1e-4), F(eps)),
        "llt": lambda f, o, it, eps, i, s: call("cilreg_llt_rof_dev", f, o, i, s, F(0.02), F(0.01), I(it), F(1e-3), F(eps)),
        "dtv": dtv,
    }


OPS = ["rof", "fgp", "pd", "sb", "tgv", "ndf", "d4", "llt", "dtv"]


def _image(shape, seed=3):
    import torch

    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0 : shape[0], 0 : shape[1]]
    img = ((x // 9 + y // 7) % 3) * 0.4 + rng.normal(0, 0.05, shape)
    return torch.from_numpy(img.astype(np.float32)).cuda()


@pytest.mark.parametrize("setting", ["1", "0"], ids=["strips", "one-iteration"])
@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", [(77, 130), (61, 91)])
def test_input_of_a_kernel_that_triggers_early(late_copy, monkeypatch, op, shape, setting):
    import torch

    monkeypatch.setenv("CILREG_STRIP2D", setting)
    call = _dev_calls()[op]
    if op == "dtv":
        call.ref = _image(shape, 4)
    img, info = _image(shape), np.zeros(2, np.float32)
    f = torch.full(shape, 7.0, device="cuda")
    out, want = torch.zeros_like(f), torch.zeros_like(f)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        s = torch.cuda.current_stream().cuda_stream
        call(img, want, 12, 0.0, info, s)
        late_copy(img, f)
        call(f, out, 12, 0.0, info, s)
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("setting", ["1", "0"], ids=["strips", "one-iteration"])
@pytest.mark.parametrize("alg,prm", [(0, [0.02, 0.001]), (1, [0.05, 0, 0]), (2, [0.05, 0]), (3, [0.02, 0.05, 0.01, 1])])
def test_prox_input_of_a_kernel_that_triggers_early(late_copy, monkeypatch, alg, prm, setting):
    import torch
    from ccpi.filters.utils import cilregcuda as C

    monkeypatch.setenv("CILREG_STRIP2D", setting)
    ny, nx = 77, 130
    img = _image((ny, nx))
    outs = []
    with torch.cuda.stream(torch.cuda.Stream()):
        s = torch.cuda.current_stream().cuda_stream
        for late in (False, True):
            h = ctypes.c_void_p()
            assert C.cilreg_prox_session_create(ctypes.byref(h), alg, (ctypes.c_float * 4)(*prm), 4, nx, ny, 1, s) == 0
            out = torch.zeros_like(img)
            for _ in range(2):  # cold, then warm
                f = img if not late else torch.full_like(img, 7.0)
                torch.cuda.synchronize()
                if late:
                    late_copy(img, f)
                assert C.cilreg_prox_session_prox(h, f.data_ptr(), out.data_ptr(), 9, 0.0, None, s) == 0
            outs.append(out)
            assert C.cilreg_prox_session_destroy(h, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("op", OPS)
def test_nothing_is_left_to_write_when_a_stopped_call_returns(op):
    """The rule fires at its fourth check (iteration 15) of 200 iterations; the
    image is large enough for a late copy to be seen still running."""
    import torch

    f = torch.rand((8192, 8192), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    call = _dev_calls()[op]
    if op == "dtv":
        call.ref = f.flip(0).contiguous()
    out, info = torch.zeros_like(f), np.zeros(2, np.float32)
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    call(f, out, 200, 1e3, info, stream.cuda_stream)
    done = stream.query()
    with torch.cuda.stream(other):
        seen = out.clone()
    torch.cuda.synchronize()
    assert int(info[0]) == 15
    assert done and torch.equal(seen, out)


@pytest.mark.parametrize("alg,prm,tol", [(1, [0.05, 0, 0], 1e3), (2, [0.05, 0], 1e3), (2, [0.05, 0], 0.0)])
def test_nothing_is_left_to_write_when_a_prox_call_returns(alg, prm, tol):
    import torch
    from ccpi.filters.utils import cilregcuda as C

    f = torch.rand((8192, 8192), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    out, info = torch.zeros_like(f), (ctypes.c_float * 2)()
    stream, h = torch.cuda.Stream(), ctypes.c_void_p()
    ny, nx = f.shape
    torch.cuda.synchronize()
    s = stream.cuda_stream
    assert C.cilreg_prox_session_create(ctypes.byref(h), alg, (ctypes.c_float * 4)(*prm), len(prm), nx, ny, 1, s) == 0
    assert C.cilreg_prox_session_prox(h, f.data_ptr(), out.data_ptr(), 100, tol, info, s) == 0
    done = stream.query()
    torch.cuda.synchronize()
    assert C.cilreg_prox_session_destroy(h, s) == 0
    assert info[0] == (15 if tol else 100)
    assert done
