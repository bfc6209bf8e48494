"""The native front of `matmul`: what it takes, what it leaves to the Python checks, and the workspaces it uses."""

import ctypes
import subprocess
import threading
import types
import weakref

import pytest
import torch

import tuna_b200
from oracle import tuna_oracle as orc
from tests.gpu_util import check_parity, make_case
from tuna_b200 import _lib, build, ops

M, N, K = 64, 3, 128


def _args(device):
    return {"x": torch.zeros((N, K), dtype=torch.float16, device=device), "q": torch.zeros((M // 8, K // 8, 32), dtype=torch.uint8, device=device),
            "s": torch.ones(M, device=device), "c": torch.linspace(-1, 1, 16, device=device),
            "o": torch.empty((N, M), dtype=torch.float16, device=device), "m": M, "n": N, "k": K}


def test_leaves_everything_unusual_to_python():
    call = _lib.load_fast_call().matmul
    a = _args("cpu")
    for args in ((), (1, 2, 3, 4, 5, 6, 7, 8), tuple(a.values()), (*list(a.values())[:5], 1 << 70, 3, 8), (*list(a.values())[:5], 64.0, 3, 128)):
        assert call(*args) is False


class _Sub(torch.Tensor):
    pass


BAD = {"cpu x": ("x", lambda t: t.cpu()), "type of x": ("x", lambda t: t.float()), "strides of x": ("x", lambda t: t.t().contiguous().t()),
       "size of q": ("q", lambda t: t[1:]), "no tensor": ("s", lambda t: 1.0), "type of c": ("c", lambda t: t.half()), "size of o": ("o", lambda t: t[:, 1:].contiguous()),
       "m": ("m", lambda v: 68), "n": ("n", lambda v: -3), "k": ("k", lambda v: 0)}


@pytest.mark.gpu
@pytest.mark.parametrize("what", BAD)
def test_bad_arguments_raise_what_the_python_checks_raise(what):
    a = _args("cuda")
    ws = tuna_b200.workspace_for(M, N, K, a["x"].device)
    tuna_b200.matmul(*a.values())  # a workspace is registered: the native way is open
    assert _lib.load_fast_call().matmul(*a.values()) is True
    name, change = BAD[what]
    a[name] = change(a[name])
    assert _lib.load_fast_call().matmul(*a.values()) is False
    raised = []
    for kw in ({}, {"workspace": ws}):  # with a workspace of its own a call takes the Python way
        with pytest.raises(Exception) as e:
            tuna_b200.matmul(*a.values(), **kw)
        raised.append((e.type, str(e.value)))
    assert raised[0] == raised[1]


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[(64, 3, 128), (4096, 17, 4104), (40000, 5, 64), (64, 3, 128)], [(512, 300, 512), (64, 1, 8)]])
def test_streams_threads_and_growing_workspaces(shapes):
    """The same GEMMs on the default stream, on two streams of their own and from threads, small shapes before large ones."""
    errors = []

    def work(stream):
        try:
            with torch.cuda.stream(stream):
                for m, n, k in shapes:
                    host, (x, q, s, c) = make_case(m, n, k, m + n)
                    for xs in (x, x.as_subclass(_Sub)):  # a subclass takes the Python way
                        o = torch.full((n, m), float("nan"), dtype=torch.float16, device="cuda")
                        tuna_b200.matmul(xs, q, s, c, o, m, n, k)
                        stream.synchronize()
                        check_parity(o.cpu().numpy(), orc.matmul_ref(*host, m, n, k), 1e-2)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    work(torch.cuda.current_stream())
    threads = [threading.Thread(target=work, args=(torch.cuda.Stream(),)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_threads_that_share_a_stream_keep_the_larger_workspace(monkeypatch):
    """A thread that meets no workspace is held up between allocating a small one and storing it; another one stores a larger one."""
    small, large, key = 2 << 20, 4 << 20, (0, 0x5EED)
    allocated, go = threading.Event(), threading.Event()
    zeros = torch.zeros

    def slow_zeros(size, **kw):
        t = zeros(size, **kw)
        if size == small:
            allocated.set()
            assert go.wait(20)
        return t

    monkeypatch.setattr(ops, "_stream_ptr", lambda device: key[1])
    monkeypatch.setattr(ops, "_workspace_bytes", lambda index, m, n, k: m)
    monkeypatch.setattr(ops.torch, "zeros", slow_zeros)
    got = []
    thread = threading.Thread(target=lambda: got.append(ops.workspace_for(small, 1, 1, "cpu:0")))
    try:
        thread.start()
        assert allocated.wait(20)
        got.append(ops.workspace_for(large, 1, 1, "cpu:0"))
        go.set()
        thread.join(20)
        assert len(got) == 2 and got[0].numel() == got[1].numel() == large
        assert got[0] is got[1] is _lib.workspaces[key]
        assert _lib.load_fast_call().workspace(*key) == (got[0].data_ptr(), large)  # what a native launch is given
        ops.workspace_for(8 << 20, 1, 1, "cpu:0")
        assert _lib.load_fast_call().workspace(*key) == (_lib.workspaces[key].data_ptr(), 8 << 20)
    finally:
        go.set()
        _lib.workspaces.pop(key, None)
    assert _lib.load_fast_call().workspace(*key) is None


@pytest.fixture
def stub():
    """Puts a function in the place of tuna_matmul: nothing is launched."""
    fast, real = _lib.load_fast_call(), ctypes.cast(_lib.load().tuna_matmul, ctypes.c_void_p).value
    yield lambda address: fast.bind(address, _lib.workspaces)
    fast.bind(real, _lib.workspaces)


@pytest.mark.gpu
def test_a_launch_holds_the_workspace_it_was_given(stub):
    a = _args("cuda")
    tuna_b200.matmul(*a.values())
    key = (0, torch.cuda.current_stream().cuda_stream)
    seen = []

    def replaced_meanwhile(*args):
        ref, size = weakref.ref(_lib.workspaces[key]), _lib.workspaces[key].numel()
        seen.append((args[8], args[9]) == (ref().data_ptr(), size))
        _lib.workspaces[key] = torch.zeros(size, dtype=torch.uint8, device="cuda")
        seen.append(ref() is not None)
        return 0

    proto = ctypes.CFUNCTYPE(ctypes.c_int, *([ctypes.c_void_p] * 5), *([ctypes.c_int] * 3), ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p)
    callback = proto(replaced_meanwhile)
    stub(ctypes.cast(callback, ctypes.c_void_p).value)
    assert _lib.load_fast_call().matmul(*a.values()) is True
    assert seen == [True, True]


@pytest.mark.gpu
def test_other_threads_run_while_a_launch_waits(stub, tmp_path):
    """A launch that waits (the stream's queue is full) for what another Python thread does."""
    src, so = tmp_path / "wait.c", tmp_path / "wait.so"
    src.write_text("#include <unistd.h>\nvolatile int entered, go;\n"
                   "int wait_for_go(void) { entered = 1; for (int i = 0; i < 500; ++i) { if (go) return 0; usleep(10000); } return 99; }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    entered, go = (ctypes.c_int.in_dll(lib, name) for name in ("entered", "go"))
    a = _args("cuda")
    tuna_b200.matmul(*a.values())
    stop = threading.Event()

    def other():
        while not entered.value and not stop.wait(0.001):
            pass
        go.value = 1

    thread = threading.Thread(target=other)
    thread.start()
    try:
        stub(ctypes.cast(lib.wait_for_go, ctypes.c_void_p).value)
        assert _lib.load_fast_call().matmul(*a.values()) is True
    finally:
        stop.set()
        thread.join()


@pytest.mark.gpu
@pytest.mark.parametrize("status,answer", [(0, True), (-4, False), (-6, -6), (-9, -9)])
def test_a_failed_call_is_not_made_again(stub, monkeypatch, status, answer):
    """Only a workspace that is too small (-4, before any launch) leaves the call to Python; a call of several passes may have launched some."""
    a = _args("cuda")
    tuna_b200.matmul(*a.values())
    calls = []
    proto = ctypes.CFUNCTYPE(ctypes.c_int, *([ctypes.c_void_p] * 5), *([ctypes.c_int] * 3), ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p)
    callback = proto(lambda *args: calls.append(args) or status)
    monkeypatch.setattr(_lib.load(), "tuna_matmul", lambda *args: pytest.fail("the Python way was taken") if status != -4 else 0)
    stub(ctypes.cast(callback, ctypes.c_void_p).value)
    assert _lib.load_fast_call().matmul(*a.values()) == answer
    if status in (0, -4):
        tuna_b200.matmul(*a.values())
    else:
        with pytest.raises(tuna_b200.TunaError) as e:
            tuna_b200.matmul(*a.values())
        assert e.value.status == status
    assert len(calls) == 2


@pytest.mark.gpu
def test_a_misaligned_slice_raises_what_the_python_way_raises():
    a = _args("cuda")
    ws = tuna_b200.workspace_for(M, N, K, a["x"].device)
    a["x"] = torch.zeros(N * K + 1, dtype=torch.float16, device="cuda")[1:].view(N, K)
    for kw in ({}, {"workspace": ws}):
        with pytest.raises(tuna_b200.TunaError) as e:
            tuna_b200.matmul(*a.values(), **kw)
        assert e.value.status == -3


def _missing():
    raise ImportError("no such module")


FRONTS = {"missing": _missing, "another torch": lambda: types.SimpleNamespace(stamp=_lib.fast_call_stamp() + "1"), "no stamp": lambda: types.SimpleNamespace()}


@pytest.fixture
def unfit_front(request, monkeypatch):
    _lib.load_fast_call.cache_clear()
    monkeypatch.setattr(_lib, "_import_fast_call", FRONTS[request.param])
    monkeypatch.setattr(ops, "_fast_matmul", ops._bind_fast_matmul)
    yield
    _lib.load_fast_call.cache_clear()


@pytest.mark.parametrize("unfit_front", FRONTS, indirect=True)
def test_without_a_front_that_fits_the_python_checks_take_the_call(unfit_front):
    a = _args("cpu")
    with pytest.warns(RuntimeWarning, match="python -m tuna_b200.build"):
        with pytest.raises(ValueError, match="must be a CUDA tensor"):
            tuna_b200.matmul(*a.values())
    assert _lib.load_fast_call() is None


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("unfit_front", FRONTS, indirect=True)
def test_matmul_without_a_front_that_fits(unfit_front):
    host, (x, q, s, c) = make_case(64, 3, 128, 1)
    o = torch.full((3, 64), float("nan"), dtype=torch.float16, device="cuda")
    tuna_b200.matmul(x, q, s, c, o, 64, 3, 128)
    check_parity(o.cpu().numpy(), orc.matmul_ref(*host, 64, 3, 128), 1e-2)


def test_the_build_makes_a_front_for_another_torch_again(monkeypatch):
    assert not build._fast_call_stale()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "1")
    assert build._fast_call_stale()
    monkeypatch.undo()
    monkeypatch.setattr(build, "FAST_CALL", build.FAST_CALL.with_name("_fast_call.none.so"))
    assert build._fast_call_stale()


def test_the_build_does_without_a_front_that_cannot_be_built(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(build, "FAST_CALL", tmp_path / "_fast_call.so")
    monkeypatch.setenv("CXX", "false")
    build._build_fast_call(False)
    assert not build.FAST_CALL.exists() and "not built" in capsys.readouterr().err
