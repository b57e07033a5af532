"""The native host path (`_lqhost`) serves plain calls and leaves every other to the Python that checks, raises or handles it."""
import os
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_what_is_not_plain_is_left_to_python():
    from latentq_llm_b200 import _lqhost as h, ops
    x, w, s = torch.zeros(4, 128, dtype=torch.bfloat16), torch.zeros(64 * 64, dtype=torch.int8), torch.zeros(64, dtype=torch.bfloat16)
    x8 = torch.zeros(4, 128, dtype=torch.int8)
    for r in (h.w4_gemm(False, x, w, s, s, None, 64, 128, 128, None, 0), h.w4_gemm(True, None, w, s, s, None, 64, 128, 128, None, 0),
              h.a8w8_gemm(x8, x8, None, None, 1.0, None, None, 0), h.a8w8_module(x8, x8, None, 1.0, None, s, None, 0),
              h.act_quant_per_token(x), h.act_quant_per_tensor(3), h.i8_dequant(x8, None, None)):
        assert r is None                                             # CPU tensors, no tensors
    with pytest.raises(TypeError):
        h.act_quant_per_token()
    with pytest.raises(TypeError):
        h.w4_gemm(False, x)
    for call in (lambda: ops.gemm_a16w4_fwd(x, w, s, s, None, 64, 128), lambda: ops.gemm_a16w4_dgrad(x, w, s, s, 64, 128), lambda: ops.gemm_a8w8(x8, x8),
                 lambda: ops.act_quant_per_token(x), lambda: ops.act_quant_per_tensor(x), lambda: ops.i8_dequant(x8, row_scales=s),
                 lambda: ops.act_quant_per_tensor(None)):
        with pytest.raises(ValueError):
            call()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [0, 1, 17, 300])
def test_native_and_python_paths_agree_and_refuse_alike(M, monkeypatch):
    from latentq_llm_b200 import ops
    N, K = 192, 256
    g = torch.Generator(device="cuda").manual_seed(M)
    x, dy = (torch.randn(M, c, device="cuda", generator=g).to(torch.bfloat16) for c in (K, N))
    w = torch.randint(-128, 128, (N * K // 2,), device="cuda", generator=g, dtype=torch.int8)
    s = (torch.rand(N * K // 128, device="cuda", generator=g) * 0.01).to(torch.bfloat16)
    z = torch.randint(0, 16, s.shape, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    w8 = torch.randint(-128, 128, (N, K), device="cuda", generator=g, dtype=torch.int8)
    x8 = torch.randint(-128, 128, (M, K), device="cuda", generator=g, dtype=torch.int8)
    rs, cs, qs = torch.rand(M, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g), (torch.rand(N, 1, device="cuda", generator=g) + 0.1).to(torch.bfloat16)
    one = torch.full((1,), 2.5, device="cuda")
    good = [lambda: ops.gemm_a16w4_fwd(x, w, s, z, bias, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s.view(-1, 1), z.view(-1, 1), None, N, K),
            lambda: ops.gemm_a16w4_dgrad(dy, w, s, z, N, K), lambda: ops.gemm_a8w8(x8, w8, rs, cs, 0.5, bias), lambda: ops.gemm_a8w8(x8, w8),
            lambda: ops.gemm_a8w8_module(x8, w8, one, 1.0, bias, qs), lambda: ops.gemm_a8w8_module(x8, w8, None, 0.01, None, qs),
            lambda: ops.act_quant_per_token(x), lambda: ops.act_quant_per_tensor(x) if M else (x, x), lambda: ops.i8_dequant(w8, row_scales=qs), lambda: ops.i8_dequant(x8, clampv=one)]
    bad = [lambda: ops.gemm_a16w4_fwd(x.float(), w, s, z, None, N, K), lambda: ops.gemm_a16w4_fwd(x.t().contiguous().t()[:, ::2], w, s, z, None, N, K // 2),
           lambda: ops.gemm_a16w4_fwd(x, w[:-1], s, z, None, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s.float(), z, None, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s, z, bias, N, K, group=96),
           lambda: ops.gemm_a16w4_fwd(x.cpu(), w, s, z, None, N, K), lambda: ops.gemm_a16w4_dgrad(dy, w, s, z, K, N), lambda: ops.gemm_a8w8(x8, w8[:, :128]),
           lambda: ops.gemm_a8w8_module(x8, w8, one.double(), 1.0, None, qs), lambda: ops.gemm_a8w8_module(x8, w8, None, 1.0, bias[:-1], qs),
           lambda: ops.act_quant_per_token(x[:, :100]), lambda: ops.act_quant_per_token(x.half()), lambda: ops.i8_dequant(w8, row_scales=qs[:-1]), lambda: ops.i8_dequant(w8)]

    def outcome(f):
        try:
            r = f()
        except Exception as e:                                       # noqa: BLE001
            return type(e), str(e)
        return r if isinstance(r, tuple) else (r,)

    native = [outcome(f) for f in good + bad]

    class Off:
        def __getattr__(self, name):
            return lambda *a: None
    monkeypatch.setattr(ops, "_host", Off())
    for f, a, n in zip(good + bad, native, range(100)):
        b = outcome(f)
        assert len(a) == len(b), (n, a, b)
        for u, v in zip(a, b):
            if isinstance(u, torch.Tensor):
                assert u.dtype == v.dtype and u.shape == v.shape and torch.equal(u, v), n
            else:
                assert u == v, (n, a, b)


# A process in which the functions that `_lqhost` calls are stand-ins that wait and return a given status (loaded first and globally, so that
# the module binds to them; `_lib`, which looks its functions up in the library itself, does not).
_STAND_IN = """
#include <unistd.h>
static int status, wait_us;
void stand_in(int s, int us) { status = s; wait_us = us; }
#define F(name) int name() { usleep(wait_us); return status; }
F(lq_gemm_a16w4_fwd) F(lq_gemm_a16w4_dgrad) F(lq_gemm_a8w8) F(lq_gemm_a8w8_module) F(lq_act_quant_per_token) F(lq_act_quant_per_tensor) F(lq_i8_dequant)
"""
_CALLS = """
import ctypes, sys, threading, time
lib = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
import torch
from latentq_llm_b200 import _lib, ops
x = torch.zeros(20, 128, dtype=torch.bfloat16, device="cuda")
w, s = torch.zeros(128 * 64, dtype=torch.int8, device="cuda"), torch.ones(128, dtype=torch.bfloat16, device="cuda")
x8, w8, one = torch.zeros(20, 128, dtype=torch.int8, device="cuda"), torch.zeros(64, 128, dtype=torch.int8, device="cuda"), torch.ones(1, device="cuda")
calls = dict(fwd=lambda: ops.gemm_a16w4_fwd(x, w, s, s, None, 128, 128), dgrad=lambda: ops.gemm_a16w4_dgrad(x, w, s, s, 128, 128), a8w8=lambda: ops.gemm_a8w8(x8, w8),
             module=lambda: ops.gemm_a8w8_module(x8, w8, one, 1.0, None, s[:64]), per_token=lambda: ops.act_quant_per_token(x),
             per_tensor=lambda: ops.act_quant_per_tensor(x), dequant=lambda: ops.i8_dequant(x8, clampv=one))
for f in calls.values():
    f()
"""


def _run_with_stand_in(tmp_path, body):
    c, so = tmp_path / "stand_in.c", tmp_path / "stand_in.so"
    c.write_text(_STAND_IN)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(so), str(c)])
    r = subprocess.run([sys.executable, "-c", _CALLS + body, str(so)], cwd=ROOT, capture_output=True, text=True, timeout=180)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.gpu
def test_other_threads_run_during_a_native_call(tmp_path):
    """A launch may wait for a full queue, an allocation for the device: what ends the wait may be another Python thread's work."""
    _run_with_stand_in(tmp_path, """
ticks, stop = [], threading.Event()
def tick():
    while not stop.wait(0.002):
        ticks.append(time.perf_counter())
t = threading.Thread(target=tick, daemon=True)
t.start()
lib.stand_in(0, 200000)
for name, f in calls.items():
    a = time.perf_counter()
    f()
    b = time.perf_counter()
    assert b - a > 0.19, (name, b - a)                               # the native function was the one that ran
    n = sum(a < u < b for u in ticks)
    assert n > 10, (name, n)
stop.set()
t.join()
""")


@pytest.mark.gpu
def test_an_error_behind_a_launch_is_raised_and_the_call_not_repeated(tmp_path):
    """What the library refuses before it launches goes to the Python, which repeats the call; any other status is an error at once."""
    _run_with_stand_in(tmp_path, """
for status in (_lib.LQ_ECUDA, _lib.LQ_ETIMEOUT, -77):
    lib.stand_in(status, 0)
    for name, f in calls.items():
        try:
            f()
        except _lib.LatentQError as e:
            assert e.status == status and str(e).startswith("lq_"), (name, e)
        else:
            raise AssertionError((name, status))
for status in (_lib.LQ_EINVAL, _lib.LQ_EUNSUPPORTED, _lib.LQ_EWORKSPACE):
    lib.stand_in(status, 0)
    y = {name: f() for name, f in calls.items()}
    torch.cuda.synchronize()
    assert all(float(y[k].float().abs().max()) == 0.0 for k in ("fwd", "dgrad", "a8w8", "module", "dequant")), status
""")


@pytest.mark.parametrize("how,says", [("sys.modules['latentq_llm_b200._lqhost'] = None", "missing or does not load"),
                                      ("import types; m = types.ModuleType('latentq_llm_b200._lqhost'); m.__file__ = 'x.so'; sys.modules[m.__name__] = p._lqhost = m", "built for torch"),
                                      ("import torch; from latentq_llm_b200 import _lqhost; _lqhost.torch_build = '2.0.0 0'", "built for torch 2.0.0 0")])
def test_a_missing_or_foreign_module_is_refused_with_the_command_to_build_it(how, says):
    """The module holds torch's inline accessors: under another torch it does not load, or reads wrong fields."""
    r = subprocess.run([sys.executable, "-c", f"import sys, latentq_llm_b200 as p; {how}\nfrom latentq_llm_b200 import ops"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 1 and says in r.stderr and "python -m latentq_llm_b200.build" in r.stderr.splitlines()[-1], r.stderr[-1000:]


def test_another_torch_makes_the_module_stale(monkeypatch):
    from latentq_llm_b200 import _lqhost, build
    assert _lqhost.__file__ == build.HOST and not build._host_stale()
    monkeypatch.setattr(torch, "__version__", "2.0.0")
    assert build._host_stale()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 17, 300])
def test_plain_calls_are_served_by_the_native_functions(M, monkeypatch):
    """Each plain call is answered by its native function, not by the Python behind it; what that refuses too raises."""
    from latentq_llm_b200 import ops
    N, K = 192, 256
    x, dy = (torch.randn(M, c, device="cuda").to(torch.bfloat16) for c in (K, N))
    w, s = torch.zeros(N * K // 2, dtype=torch.int8, device="cuda"), torch.ones(N * K // 128, 1, dtype=torch.bfloat16, device="cuda")
    x8, w8, qs, one = torch.zeros(M, K, dtype=torch.int8, device="cuda"), torch.zeros(N, K, dtype=torch.int8, device="cuda"), s[:N], torch.ones(1, device="cuda")
    bias = qs.view(-1)
    served = []

    class Recorder:
        def __getattr__(self, name):
            def f(*a, _native=getattr(native, name)):
                r = _native(*a)
                served.append((name, r is not None))
                return r
            return f
    native = ops._host
    monkeypatch.setattr(ops, "_host", Recorder())
    for name, call in (("w4_gemm", lambda: ops.gemm_a16w4_fwd(x, w, s, s, bias, N, K)), ("w4_gemm", lambda: ops.gemm_a16w4_dgrad(dy, w, s, s, N, K)),
                       ("a8w8_gemm", lambda: ops.gemm_a8w8(x8, w8, torch.ones(M, device="cuda"), None, 1.0, bias)), ("a8w8_module", lambda: ops.gemm_a8w8_module(x8, w8, one, 1.0, bias, qs)),
                       ("act_quant_per_token", lambda: ops.act_quant_per_token(x)), ("act_quant_per_tensor", lambda: ops.act_quant_per_tensor(x)),
                       ("i8_dequant", lambda: ops.i8_dequant(w8, row_scales=qs)), ("i8_dequant", lambda: ops.i8_dequant(x8, clampv=one))):
        served.clear()
        assert call() is not None and served == [(name, True)], (name, served)
    for call in (lambda: ops.gemm_a16w4_fwd(x.float(), w, s, s, None, N, K), lambda: ops.gemm_a16w4_fwd(x, w, s, s, None, N, K, group=96),
                 lambda: ops.gemm_a8w8(x8, w8[:, :128]), lambda: ops.gemm_a8w8_module(x8, w8, None, 1.0, bias[:-1], qs), lambda: ops.act_quant_per_token(x[:, :100]),
                 lambda: ops.act_quant_per_tensor(x.half()), lambda: ops.i8_dequant(w8, row_scales=qs[:-1])):
        served.clear()
        with pytest.raises(Exception):
            call()
        assert not any(ok for _, ok in served)


class _OnGpu:
    """What `linear_rows` may ask of a CUDA tensor, without one."""

    def __init__(self, *shape, at=0, index=0, dtype=torch.bfloat16, cuda=True, contiguous=True, grad=False):
        self.shape, self.at, self.dtype, self.is_cuda, self.requires_grad, self._contiguous = torch.Size(shape), at, dtype, cuda, grad, contiguous
        self.device = torch.device("cuda", index) if cuda else torch.device("cpu")

    def is_contiguous(self):
        return self._contiguous

    def data_ptr(self):
        return self.at

    def dim(self):
        return len(self.shape)

    def numel(self):
        return self.shape.numel()

    def copy_(self, y):
        return self


def test_linear_rows_gives_the_kernel_nothing_that_it_may_not_touch(monkeypatch):
    """Which calls reach the library's entry (a stub here) and which torch's linear, which moves, records or refuses as it always does."""
    from types import SimpleNamespace

    from latentq_llm_b200 import ops
    monkeypatch.setattr(torch, "Tensor", _OnGpu)                     # (the stand-ins count as plain tensors)
    went = []
    monkeypatch.setattr(ops.L, "lib", SimpleNamespace(lq_linear_rows=lambda *a: (went.append("kernel"), 0)[1]))
    monkeypatch.setattr(torch.nn.functional, "linear", lambda x, w: (went.append("torch"), _OnGpu(1))[1])
    monkeypatch.setattr(torch, "empty", lambda shape, dtype=None, device=None: _OnGpu(*shape, at=1 << 40))
    monkeypatch.setattr(ops, "_current_device", lambda: 0)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    M, N, K, mib = 4, 100, 4096, 1 << 20

    def route(x=None, w=None, out=None, **ctx):
        went.clear()
        ops.linear_rows(x or _OnGpu(M, K, at=mib), w or _OnGpu(N, K, at=2 * mib), out)
        return went

    assert route() == ["kernel"] and route(out=_OnGpu(M, N, at=16 * mib)) == ["kernel"]
    assert route(out=_OnGpu(M, N, at=mib + 2 * M * K)) == ["kernel"] and route(out=_OnGpu(M, N, at=mib - 2 * M * N)) == ["kernel"]     # side by side
    for case in (dict(out=_OnGpu(M, N, at=16 * mib, cuda=False)), dict(out=_OnGpu(M, N, at=16 * mib, index=1)), dict(w=_OnGpu(N, K, at=2 * mib, index=1)),
                 dict(w=_OnGpu(N, K, at=2 * mib, cuda=False)), dict(x=_OnGpu(M, K, at=mib, index=1), w=_OnGpu(N, K, at=2 * mib, index=1)),     # not the current device
                 dict(out=_OnGpu(M, N, at=mib)), dict(out=_OnGpu(M, N, at=mib + 2 * M * K - 2)), dict(out=_OnGpu(M, N, at=mib - 2 * M * N + 2)),
                 dict(out=_OnGpu(M, N, at=2 * mib + 64)), dict(out=_OnGpu(N, M, at=16 * mib)), dict(out=_OnGpu(M, N, at=16 * mib, dtype=torch.float32)),
                 dict(x=_OnGpu(9, K, at=mib)), dict(x=_OnGpu(0, K, at=mib)), dict(x=_OnGpu(M, K, at=mib + 2)), dict(w=_OnGpu(N, K, at=2 * mib, contiguous=False)),
                 dict(w=_OnGpu(N, 2048, at=2 * mib)), dict(x=_OnGpu(M, K, at=mib, grad=True)), dict(w=_OnGpu(N, K, at=2 * mib, grad=True)),
                 dict(x=_OnGpu(2, 2, K, at=mib))):
        assert route(**case) == ["torch"], vars(next(iter(case.values())))
    with torch.no_grad():
        assert route(w=_OnGpu(N, K, at=2 * mib, grad=True)) == ["kernel"]
        with torch.autograd.forward_ad.dual_level():
            assert route() == ["torch"]
