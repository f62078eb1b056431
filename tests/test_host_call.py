"""The way from Python to the launchers: arguments arrive as ctypes would pass them, outputs are torch.empty's."""
import ctypes
import shutil
import subprocess
import threading
from types import SimpleNamespace

import pytest
import torch

from questwend_b200.kernels import build, ops

SOURCE = """
#include <string.h>
static unsigned char seen[512];
int take(void* a, int b, float c, double d, long long e, void* g, int h, int i, int j, unsigned k, float l, unsigned long long m, int n, float o, void* p, int q) {
    unsigned char* s = seen;
#define KEEP(x) memcpy(s, &x, sizeof x); s += sizeof x
    KEEP(a); KEEP(b); KEEP(c); KEEP(d); KEEP(e); KEEP(g); KEEP(h); KEEP(i); KEEP(j); KEEP(k); KEEP(l); KEEP(m); KEEP(n); KEEP(o); KEEP(p); KEEP(q);
    return (int)(s - seen);
}
int refuse(void) { return -7; }
void* what(void) { return seen; }
"""


@pytest.fixture(scope="module")
def host():
    if not shutil.which("g++") and not build.host_calls_built():
        pytest.skip("no g++")
    build.compile_host_calls()
    module = build.host_calls()
    assert module is not None
    return module


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not shutil.which("gcc"):
        pytest.skip("no gcc")
    d = tmp_path_factory.mktemp("c")
    (d / "take.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", str(d / "take.so"), str(d / "take.c")], check=True)
    lib = ctypes.CDLL(str(d / "take.so"))
    lib.what.restype = ctypes.c_void_p
    return lib


def test_arguments_arrive_as_through_ctypes(host, lib):
    t, u = torch.arange(6.0)[2:], torch.zeros(3, dtype=torch.bfloat16)
    address = lambda name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value
    n = lib.take(ctypes.c_void_p(t.data_ptr()), ctypes.c_int(-3), ctypes.c_float(1e-6), ctypes.c_double(-2.25), ctypes.c_longlong(-(2 ** 40)), ctypes.c_void_p(0), ctypes.c_int(1),
                 ctypes.c_int(2 ** 31 - 1), ctypes.c_int(0), ctypes.c_uint(2 ** 32 - 5), ctypes.c_float(0.1), ctypes.c_ulonglong(2 ** 64 - 2), ctypes.c_int(9),
                 ctypes.c_float(-0.0), ctypes.c_void_p(u.data_ptr()), ctypes.c_int(77))
    want = ctypes.string_at(lib.what(), n)
    ctypes.memset(lib.what(), 0, n)
    args = (t, -3, 1e-6, ctypes.c_double(-2.25), ctypes.c_longlong(-(2 ** 40)), None, True, 2 ** 31 - 1, False, ctypes.c_uint(2 ** 32 - 5), 0.1, ctypes.c_ulonglong(2 ** 64 - 2), 9,
            ctypes.c_float(-0.0), torch.nn.Parameter(u, requires_grad=False), 77)
    assert host.call(address("take"), *args) == n and ctypes.string_at(lib.what(), n) == want
    assert host.call(address("refuse")) == -7
    for bad in (("x",), ([1],), (1j,), tuple(range(57)), (0.5,) * 9):
        with pytest.raises((TypeError, AttributeError)):
            host.call(address("refuse"), *bad)
    with pytest.raises(ValueError):
        host.call(0)


def test_tensors_that_fit_and_outputs(host):
    assert not host.fits(torch.zeros(2), torch.float32, 1) and not host.fits(None, None, None) and not host.fits("x", None, 1)      # none on a GPU
    for shape, dtype in (((2, 3), torch.bfloat16), ((), torch.int32), ((0, 5), torch.float64), (4, torch.uint8), ([2, 2], torch.float32)):
        for device in (torch.device("cpu"), "cpu"):
            t = host.empty(shape, dtype=dtype, device=device)
            want = torch.empty(shape, dtype=dtype, device=device)
            assert t.shape == want.shape and t.dtype == dtype and t.device == want.device and t.is_contiguous() and not t.requires_grad
    for bad in (dict(dtype=torch.float32, device="nowhere"), dict(dtype=3, device="cpu")):
        with pytest.raises((TypeError, RuntimeError)):
            host.empty((2,), **bad)
    with pytest.raises(RuntimeError):
        host.empty((-1,), dtype=torch.float32, device=torch.device("cpu"))
    x = object()
    assert host.same(x) is x


def test_lists_into_arrays(host):
    import numpy as np
    a = np.zeros(5, dtype=np.int32)
    assert host.fill(a[1:4], [2 ** 31 - 1, -(2 ** 31), 7]) and a.tolist() == [0, 2 ** 31 - 1, -(2 ** 31), 7, 0] and host.fill(a[:0], [])
    for array, numbers in ((a, [1, 2]), (a[:2], (1, 2)), (a[:2], [1, 2.0]), (a[:2], [1, True]), (a[:2], [1, 2 ** 31]), (a[:2], [1, -(2 ** 80)]), (a[:2], [1, np.int32(2)]),
                           (np.zeros(2, dtype=np.int64), [1, 2]), (np.zeros(2, dtype=np.float32), [1, 2])):
        assert host.fill(array, numbers) is False
    with pytest.raises((BufferError, ValueError)):
        host.fill(np.zeros(4, dtype=np.int32)[::2], [1, 2])


def test_a_launcher_is_looked_up_by_several_threads_at_once(host, lib, monkeypatch):
    """A thread that finds another one in the middle of the first look-up of a launcher."""
    others, errors = [], []

    def call():
        try:
            ops._call("module", "take", *range(16))
        except Exception as e:          # noqa: BLE001 - reported below
            errors.append(e)

    def cast(*args):
        if not others:
            others.append(threading.Thread(target=call))
            others[0].start()
            others[0].join()
        return ctypes.cast(*args)

    monkeypatch.setattr(ops, "_HOST", SimpleNamespace(call=lambda address, *args: 0))
    monkeypatch.setattr(ops, "load_module", lambda name: lib)
    monkeypatch.setattr(ops, "ctypes", SimpleNamespace(cast=cast, c_void_p=ctypes.c_void_p))
    monkeypatch.setattr(ops, "_FUNCTIONS", {})
    monkeypatch.setattr(ops, "_ADDRESSES", {})
    call()
    assert others and not errors, errors


@pytest.fixture
def unbound(monkeypatch):
    """As in a process that has not looked a launcher up, where the native module was not there at the import."""
    for name in ("_HOST", "_ptr", "_i", "_f", "_address", "_empty"):
        monkeypatch.setattr(ops, name, getattr(ops, name))
    monkeypatch.setattr(ops, "_host_wanted", True)
    monkeypatch.setattr(build, "_host_loaded", [])
    ops._bind_host(None)


def test_the_native_module_is_built_on_first_use(host, lib, unbound, tmp_path, monkeypatch):
    built = build._host_path()
    monkeypatch.setattr(build, "_host_path", lambda: str(tmp_path / "qwb_host_call.so"))
    monkeypatch.setattr(build, "_host_command", lambda out: ["cp", built, out])         # what g++ would write
    monkeypatch.setattr(ops, "load_module", lambda name: lib)
    monkeypatch.setattr(ops, "_FUNCTIONS", {})
    monkeypatch.setattr(ops, "_ADDRESSES", {})
    assert not build.host_calls_built()
    args = (ops._ptr(None), ops._i(-3), ops._f(0.5), ctypes.c_double(1.5), ctypes.c_longlong(7), ops._ptr(torch.zeros(1)), *(ops._i(i) for i in range(3)), ctypes.c_uint(9),
            ops._f(2.0), ctypes.c_ulonglong(3), ops._i(4), ops._f(1.0), ops._address(64), ops._i(5))
    n = lib.take(*args)
    want = ctypes.string_at(lib.what(), n)
    with pytest.raises(AttributeError):                     # of the library, behind the look-up; made for ctypes, these go either way
        ops._call("module", "take", *args)
    assert build.host_calls_built() and ops._HOST is not None and ops._i(3) == 3 and ops._empty is ops._HOST.empty
    assert ctypes.string_at(lib.what(), n) == want
    assert ops.fill_int32(torch.zeros(2, dtype=torch.int32).numpy(), [1, 2])


def test_without_a_compiler_calls_go_through_ctypes(unbound, tmp_path, monkeypatch, capfd):
    monkeypatch.setattr(build, "_host_path", lambda: str(tmp_path / "qwb_host_call.so"))
    for command in (["false"], [str(tmp_path / "no-such-compiler")]):
        monkeypatch.setattr(build, "_host_loaded", [])
        monkeypatch.setattr(build, "_host_command", lambda out: command)
        build.compile_modules([])                           # says so and goes on
        assert build.host_calls() is None and capfd.readouterr().err.count("through ctypes") == 1
        with pytest.raises(build.KernelBuildError):
            build.compile_host_calls()
    ops._bind_host(build.host_calls())
    assert ops._HOST is None and ops._empty is torch.empty and not ops.fill_int32(torch.zeros(1, dtype=torch.int32).numpy(), [1])


@pytest.mark.gpu
def test_kernels_through_both_ways_give_the_same_bits(host, unbound):
    dev = torch.device("cuda:0")
    torch.manual_seed(1)
    x, w = torch.randn(9, 256, device=dev), 1 + torch.rand(256, device=dev)
    xb, wb = x.bfloat16(), torch.randn(64, 256, device=dev).bfloat16()
    positions, freq = torch.arange(9, device=dev).int(), torch.rand(32, device=dev, dtype=torch.float64)
    chosen, weight = torch.randint(0, 8, (9, 2), device=dev).int(), torch.rand(9, 2, device=dev)
    up, down = torch.randn(8, 16, 256, device=dev), torch.randn(8, 256, 16, device=dev)

    def run():
        return [ops.rmsnorm(x, w, 1e-6, torch.float32), ops.gemm_tc(xb, wb), *ops.rope_table(positions, freq, 0.75), *ops.moe_route(x[:, :8].contiguous(), 2, weight_scale=0.3),
                ops.moe_experts(x, up, down, chosen, weight, "relu2"), ops.sample(x, 0.8, top_k=5, top_p=0.9, seed=3)]

    results = []
    for module in (None, host):
        ops._bind_host(module)
        results.append(run())
    assert all(torch.equal(a, b) for a, b in zip(*results))
    with pytest.raises(ops.KernelError, match="weight has"):
        ops.rmsnorm(x, w[:8].contiguous(), 1e-6, torch.float32)
