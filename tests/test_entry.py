"""The module that calls the kernel library's entry points (csrc/host/entry.cpp): its reading of arguments and tensors."""
import itertools

import pytest
import torch

from dotllm_b200.errors import KernelError
from dotllm_b200.kernels import gemm_skinny, library


@pytest.fixture(scope="module")
def entry():
    return library.entry()


def test_every_declared_entry_point_is_bound_with_its_own_arguments(entry):
    for name in library._SIGNATURES:
        assert callable(library._bind(name))


def test_declarations_that_differ_from_the_library_are_refused(entry, monkeypatch):
    monkeypatch.setitem(library._SIGNATURES, "dl_add_rows", library._SIGNATURES["dl_add_rows"] + [library._I])
    with pytest.raises(KernelError, match="declared"):
        library._bind("dl_add_rows")
    assert entry.bind(entry.handle, "dl_no_such_thing") is None


def test_arguments(entry):
    pieces = library._bind("dl_chunk_pieces")
    assert pieces(100, 3) == (100 + 31 * 3) // 32
    assert pieces(True, 2**32 + 3) == (1 + 31 * 3) // 32         # as ctypes: the low 32 bits
    for bad in ((1,), (1, 2, 3)):
        with pytest.raises(TypeError):
            pieces(*bad)
    for bad in (1.5, "1", None, torch.zeros(1)):
        with pytest.raises(TypeError):
            pieces(1, bad)
    # a float where a pointer belongs, and a text where a float does
    with pytest.raises(TypeError):
        library._bind("dl_scale_values")(1.0, 1, 1.0, None)
    with pytest.raises(TypeError):
        library._bind("dl_scale_values")(None, 1, "x", None)
    with pytest.raises(KernelError, match="dl_scale_values"):        # a status becomes the library's own error
        library.call("dl_scale_values", None, -1, 1.0, None)


def test_row_stride_is_that_of_the_python_rule(entry):
    base = torch.zeros(6, 8)
    views = [base, base[:, 2:5], base[:1], base[:1, :3], base[:, :1], base[::2], base.t(), base[:, ::2], base[0], base[:0], base[:, :0], base.view(2, 3, 8),
             base.t()[:, :1], base[:1, ::2], torch.zeros(1, 1), torch.zeros(4, 1).t()]
    for t in views:
        if t.dim() != 2 or (t.shape[1] > 1 and t.stride(1) != 1):
            expected = -1
        else:
            expected = t.stride(0) if t.shape[0] > 1 else max(t.stride(0), t.shape[1])
        assert entry.row_stride(t) == expected, (t.shape, t.stride())
    assert entry.row_stride(3) == -1


def test_tensors_without_a_gpu(entry):
    x = torch.zeros(2, 8)
    assert entry.product(x, x) is None and not entry.all_cuda(x) and entry.all_cuda(None)
    for half, dtype in ((False, torch.float32), (True, torch.bfloat16)):
        t = entry.empty(3, 5, half, x)
        assert t.shape == (3, 5) and t.dtype == dtype and t.is_contiguous() and not t.is_cuda
    with pytest.raises((RuntimeError, TypeError)):
        entry.empty(-1, 5, False, x)
    assert library.empty(2, 3, torch.int32, x).dtype == torch.int32


@pytest.mark.parametrize("lacking", ["compiler", "Python.h", "broken"])
def test_machines_without_the_modules_headers_call_by_ctypes(entry, lacking, monkeypatch, tmp_path, capsys):
    """The kernel library alone is enough to run: where the module cannot be built, the missing piece is named and the calls go through ctypes."""
    import sysconfig
    from dotllm_b200.kernels import build
    monkeypatch.setattr(library, "_entry", None)
    monkeypatch.setattr(library, "_callables", {})
    monkeypatch.setattr(build, "ENTRY", "dotllm_entry_of_a_test")
    monkeypatch.setattr(build, "build_dir", lambda: tmp_path)
    if lacking == "compiler":
        monkeypatch.delenv("CXX", raising=False)
        monkeypatch.setattr(build.shutil, "which", lambda name: None)
    elif lacking == "Python.h":
        paths = sysconfig.get_paths()
        monkeypatch.setattr(sysconfig, "get_paths", lambda *a: {**paths, "include": str(tmp_path)})
    else:
        monkeypatch.setenv("CXX", "/bin/false")
    pieces = library._bind("dl_chunk_pieces")
    assert isinstance(library.entry(), library._CtypesEntry) and {"compiler": "C++ compiler", "Python.h": "Python.h", "broken": "failed"}[lacking] in capsys.readouterr().err
    assert pieces(100, 3) == entry.bind(entry.handle, "dl_chunk_pieces")(100, 3)
    for bad in ((1,), (1, 2, 3), (1, 1.5), (1, "1"), (1, None), (1, torch.zeros(1))):
        with pytest.raises(TypeError):
            pieces(*bad)
    for name in library._SIGNATURES:
        assert callable(library._bind(name))
    with pytest.raises(KernelError, match="dl_scale_values"):
        library.call("dl_scale_values", None, -1, 1.0, None)
    assert library.empty(2, 3, torch.bfloat16, torch.zeros(1)).dtype == torch.bfloat16


@pytest.mark.gpu
def test_kernels_called_by_ctypes_give_the_same(entry, monkeypatch):
    from dotllm_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    x, w = (torch.randn(*s, generator=g).to(torch.bfloat16).cuda() for s in ((5, 520), (96, 520)))
    x32, gain = x.float(), torch.rand(520, generator=g).cuda()

    def run():
        return [ops.linear(x, w), ops.gated_linear(x, w), ops.linear(x32, w.float()), ops.add_rmsnorm(x32.clone(), None, gain, 1e-5, torch.bfloat16),
                ops.linear(x[:, 8:264], w[:, :256].contiguous(), out_dtype=torch.float32)]

    want = run()
    torch.cuda.synchronize()
    monkeypatch.setattr(library, "_entry", library._CtypesEntry())
    monkeypatch.setattr(library, "_callables", {})
    library._entry.handle = None
    with torch.cuda.stream(torch.cuda.Stream()):
        got = run()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    with pytest.raises(KernelError):
        ops.linear(x, w[:, :256].contiguous())
    with pytest.raises(KernelError):
        ops.linear(x.cpu(), w)


def test_allocation_leaves_other_threads_running(entry):
    """``empty`` gives up the interpreter's lock: another thread runs although the interpreter itself would not switch for a minute."""
    import _thread
    import sys
    like, ran, kept = torch.zeros(1), [], []
    before = sys.getswitchinterval()
    sys.setswitchinterval(60.0)
    try:
        _thread.start_new_thread(lambda: ran.append(1), ())  # (threading's start() waits for the thread, and gives up the lock itself)
        for _ in range(3000):                                # (kept: a tensor's end may give up the lock as well)
            kept.append(entry.empty(512, 512, False, like))
            if ran:
                break
        assert ran
    finally:
        sys.setswitchinterval(before)


def test_every_code_that_kernels_share_has_a_text(monkeypatch):
    """A wait that ran out says in words whose it was; codes from 10 on belong to one kernel each, whose source lists them."""
    import re
    from dotllm_b200.kernels import build
    written = set()
    for source in build.sources():
        written |= {int(n) for n in re.findall(r"(?:atomicExch\(\w*\.?status, |\bgave\()(\d)\)", source.read_text())}
    assert written == set(library._STATUS_TEXT)
    for code in written:
        monkeypatch.setattr(library, "_status", {None: torch.full((1,), code, dtype=torch.int32)})
        with pytest.raises(KernelError, match="gave up: a.* (expired|pool)$"):
            library.check_status()
        library.check_status()                               # the word is clear again


@pytest.mark.gpu
def test_sizes_of_a_product_say_what_the_general_rule_says(entry):
    """``product`` against the rules it stands for, over types, strides, offsets and odd sizes."""
    big = torch.zeros(64 * 1024, device="cuda")
    for dtype, wtype in itertools.product((torch.float32, torch.bfloat16, torch.float16), (torch.float32, torch.bfloat16)):
        flat, wflat = big.to(dtype), big.to(wtype)
        for m, k, ld, at, order in itertools.product((0, 1, 2, 9, 11), (8, 12, 24), (24, 28, 32), (0, 1, 8), ("rows", "columns")):
            x = flat.as_strided((m, k), (ld, 1) if order == "rows" else (1, ld), at)
            for n, w_at in ((1, 0), (16, 0), (17, 4), (16, 8)):
                w = wflat.as_strided((n, k), (k, 1), w_at)
                got = entry.product(x, w)
                rows_ok = x.shape[1] <= 1 or x.stride(1) == 1
                if dtype != wtype or dtype == torch.float16 or not rows_ok:
                    assert got is None
                    continue
                assert got[:4] == (m, k, n, x.stride(0) if m > 1 else max(x.stride(0), k))
                if dtype == torch.float32:
                    assert got[4] == 0
                elif 1 <= m <= gemm_skinny.SKINNY_ROWS:
                    assert (got[4] == 2) == gemm_skinny.takes(x, w), (m, k, ld, at, n, w_at)
            assert entry.product(x, wflat.as_strided((16, k + 8), (k + 8, 1))) is None
            assert entry.product(x, wflat.as_strided((16, k), (1, 16))) is None        # not contiguous
