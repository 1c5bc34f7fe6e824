"""The module through which Python calls the kernels' entry points: what an entry point receives, what is refused, what is counted."""

from __future__ import annotations

import ctypes
import itertools

import pytest
import torch

from edgerag_b200.ops import kernels, native

KINDS = {ctypes.c_void_p: "p", ctypes.c_int: "i", ctypes.c_longlong: "i", ctypes.c_float: "f"}


@pytest.fixture()
def host():
    module = native.load_host()
    assert module is not None
    counts = {"own": 0, "library": 0}
    module.bind(counts, kernels.KernelError, kernels._need_in_python)
    yield module, counts
    if kernels._host:
        module = kernels._host
    module.bind(kernels.launch_counts, kernels.KernelError, kernels._need_in_python)


def _entry(host, types, result=0, own=1):
    got = []
    fn = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *a: got.append(a) or result)
    error = ctypes.CFUNCTYPE(ctypes.c_char_p)(lambda: b"what went wrong")
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value      # noqa: E731
    return host.launcher(address(fn), address(error), "".join(KINDS[t] for t in types), own), got, (fn, error)


@pytest.mark.parametrize("name", sorted(kernels._SIGNATURES))
def test_every_signature_arrives_in_order(host, name):
    types = kernels._SIGNATURES[name]
    fn, got, _keep = _entry(host[0], types)
    t = torch.arange(7.0)[3:]
    numbers = itertools.count(3)
    args = [t if k is ctypes.c_void_p and i % 3 == 0 else None if k is ctypes.c_void_p and i % 3 == 1 else
            next(numbers) / 4 if k is ctypes.c_float else -next(numbers) if k is ctypes.c_int else (1 << 40) + next(numbers)
            for i, k in enumerate(types)]
    host[0].call(fn, *args)
    assert got == [tuple(t.data_ptr() if a is t else a for a in args)]
    assert host[1] == {"own": 1, "library": 0}


@pytest.mark.parametrize("name", sorted(kernels._SIGNATURES))
def test_every_signature_arrives_without_the_module(monkeypatch, name):
    """The way through ctypes, where the module cannot be built: tensors become pointers, launches are counted, refusals raised."""
    types, got, result = kernels._SIGNATURES[name], [], [0]
    callback = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *a: got.append(a) or result[0])
    entry = ctypes.CFUNCTYPE(ctypes.c_int)(ctypes.cast(callback, ctypes.c_void_p).value)       # (as a library gives it: no types yet)
    library = type("Library", (), {name: entry, "erb_last_error": staticmethod(lambda: b"what went wrong")})
    counts = {"own": 0, "library": 0}
    for attribute, value in (("_host", False), ("_functions", {}), ("launch_counts", counts), ("_need", kernels._need_in_python)):
        monkeypatch.setattr(kernels, attribute, value)
    monkeypatch.setattr(kernels.native, "load", lambda *a: library)
    fn = kernels._fn("any", None, name)
    t, numbers = torch.arange(7.0)[3:], itertools.count(3)
    args = [t if k is ctypes.c_void_p and i % 3 == 0 else None if k is ctypes.c_void_p and i % 3 == 1 else
            next(numbers) / 4 if k is ctypes.c_float else -next(numbers) if k is ctypes.c_int else (1 << 40) + next(numbers)
            for i, k in enumerate(types)]
    call = kernels._call_in_python
    call(fn, *args)
    assert got == [tuple(t.data_ptr() if a is t else a for a in args)]
    own = kernels._LAUNCHES.get(name, 1)
    assert counts == ({"own": own, "library": 0} if own else {"own": 0, "library": 1})
    result[0] = 3
    with pytest.raises(kernels.KernelError, match="what went wrong"):
        call(fn, *args)


@pytest.mark.gpu
def test_kernels_run_without_the_module():
    """A norm, a product and decode attention in a program that has no host module: the results of one that has."""
    import multiprocessing

    context = multiprocessing.get_context("spawn")
    with context.Pool(1) as pool:
        alone = pool.apply(_run_a_few, (False,))
    assert all(a == b for a, b in zip(alone, _run_a_few(True)))


def _run_a_few(module):
    if not module:
        native.load_host = lambda: None
    g = torch.Generator().manual_seed(0)
    rand = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()       # noqa: E731
    hidden, normed = torch.randn(4, 512, generator=g).cuda(), torch.empty(4, 512, dtype=torch.bfloat16, device="cuda")
    kernels.add_rmsnorm(hidden, torch.ones(512, device="cuda"), normed, 1e-5, delta=rand(4, 512))
    q = torch.empty(4, 512, dtype=torch.bfloat16, device="cuda")
    kernels.linear(normed, rand(512, 512), q)
    pages, i32, out = rand(8, 8, 16, 64), lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda"), torch.empty_like(q)      # noqa: E731
    kernels.attention_decode_bulk(q, pages, pages, i32(0, 1, 2, 3, 4, 5, 6, 7).view(4, 2), i32(0, 1, 2, 3), i32(3, 20, 31, 8), out, 8, 0.125,
                                  torch.empty(4096, device="cuda"), torch.empty(4096, device="cuda"), 1, i32(0))
    assert (kernels._host is not False) == module
    return [t.float().cpu().tolist() for t in (hidden, normed, q, out)]


def test_results_counts_and_refusals(host):
    module, counts = host
    fn, got, _a = _entry(module, [ctypes.c_int], result=5, own=0)
    assert fn(3) == 5 and counts == {"own": 0, "library": 0}
    with pytest.raises(kernels.KernelError, match="what went wrong"):
        module.call(fn, True)
    assert counts == {"own": 0, "library": 1} and got == [(3,), (1,)]
    fn._erb_own = 2
    with pytest.raises(kernels.KernelError):
        module.call(fn, -1)
    assert counts == {"own": 2, "library": 1}
    for bad in ((), (1, 2), (1.5,), (None,), ("1",)):
        with pytest.raises(TypeError):
            module.call(fn, *bad)
    assert len(got) == 3


def test_checks_are_those_of_python(host):
    t = torch.zeros(4, 4)
    for args, kw in (((None, "x"), {}), ((t, "x"), {}), ((t, "x", torch.float32), {"contiguous": False}), ((t.t(), "x", torch.int32), {})):
        outcomes = []
        for check in (host[0].need, kernels._need_in_python):
            try:
                outcomes.append(check(*args, **kw))
            except kernels.KernelError as e:
                outcomes.append(str(e))
        assert outcomes[0] == outcomes[1]


def test_a_program_keeps_its_own_module_of_any_name(monkeypatch):
    """Loading the host module takes no name among the modules of the program."""
    import sys

    own = object()
    monkeypatch.setitem(sys.modules, "launch", own)
    before = {name: id(module) for name, module in sys.modules.items()}
    module = native.load_host()
    assert module is not None and {name: id(m) for name, m in sys.modules.items()} == before
    assert callable(module.need) and module.__name__.startswith("edgerag_b200.")


class _Silent(torch.Tensor):
    """A tensor class on a device that answers no question about its layout or memory."""

    @staticmethod
    def __new__(cls):
        return torch.Tensor._make_wrapper_subclass(cls, (4, 4), device="cuda", dtype=torch.float32, dispatch_sizes_strides_policy="strides")

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise RuntimeError(f"no answer to {func}")


def test_a_tensor_that_raises_does_not_end_the_process():
    """What torch throws behind the check or the pointer is an exception in Python (in a child: it used to abort)."""
    import multiprocessing

    child = multiprocessing.get_context("spawn").Process(target=_ask_a_silent_tensor)
    child.start()
    child.join(120)
    assert child.exitcode == 0


def _ask_a_silent_tensor():
    module = native.load_host()
    module.bind(dict.fromkeys(("own", "library"), 0), kernels.KernelError, kernels._need_in_python)
    fn, got, _keep = _entry(module, [ctypes.c_void_p])
    for ask in (lambda: kernels._need_in_python(_Silent(), "x"), lambda: module.need(_Silent(), "x"), lambda: module.call(fn, _Silent())):
        try:
            ask()
        except RuntimeError:
            continue
        assert got and got[0][0] is None, got            # (memory that is not there is a null pointer)
