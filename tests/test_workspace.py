"""The memory that the GEMM binding hands to the library: who shares it, who keeps it, what happens without it.  The parts that
need no GPU run on host tensors with a stand-in for the library."""
import contextlib
import ctypes
import threading

import numpy as np
import pytest
import torch

from oracle import oracle as O
from test_gpu_gemm import _dev, _off, make_case


class FakeLibrary:
    """Takes the GEMM calls, asks for `need` bytes and keeps (algorithm, workspace address, workspace bytes) of each."""

    def __init__(self, need, inside=lambda: None):
        self.need, self.inside, self.calls = need, inside, []

    def flh_b200_last_error(self):
        return b""

    def flh_b200_gemm_workspace_bytes(self, *a):
        return self.need

    def flh_b200_gemm_pick_algo(self, M, *a):
        return 4 if M <= 64 else 1

    def flh_b200_gemm_i4_dequant(self, *a):
        self.calls.append((a[14], a[15], a[16]))
        self.inside()
        return 0

    def flh_b200_gemm_i8w_dequant(self, *a):
        self.calls.append((None, a[12], a[13]))
        self.inside()
        return 0


@pytest.fixture
def binding(monkeypatch):
    import flh_b200
    C = flh_b200._CUDA
    monkeypatch.setattr(C, "_guard", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(C, "_stream", lambda t: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)

    def use(fake):
        monkeypatch.setattr(flh_b200._lib, "load", lambda: fake)
        return C
    return use


def _operands(m, n=128, k=256):
    return (torch.zeros(m, k // 2, dtype=torch.uint8), torch.zeros(n, k // 2, dtype=torch.uint8),
            torch.zeros(m, k // 128, dtype=torch.float16), torch.zeros(n, k // 128, dtype=torch.float16))


@pytest.mark.parametrize("entry", ["gemm_i4_dequant", "gemm_i8w_dequant"])
def test_calls_in_flight_have_scratch_of_their_own(binding, entry):
    """A prefill GEMM is two launches that meet in its scratch; two threads inside the library at once must not share it."""
    both = threading.Barrier(2, timeout=60)
    fake = FakeLibrary(4096, both.wait)
    C = binding(fake)
    A, B, SA, SB = _operands(100)
    if entry == "gemm_i8w_dequant":
        B = torch.zeros(128, 256, dtype=torch.uint8)
    threads = [threading.Thread(target=lambda: getattr(C, entry)(A, B, SA, SB)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    (_, p0, n0), (_, p1, n1) = fake.calls
    assert p0 and p1 and (p0 + n0 <= p1 or p1 + n1 <= p0)


def test_linear_refuses_zero_points_that_are_not_a_row_each(binding, monkeypatch):
    """Three tokens with one zero-point: an error, not a read past the end of the array."""
    from flh_b200.nn import LinearFLH
    fake = FakeLibrary(0)
    binding(fake)
    monkeypatch.setattr(LinearFLH, "w_rowsum", lambda self, group: torch.zeros(128, 256 // group, dtype=torch.int32))
    lin = LinearFLH(256, 128, dtype=torch.float16, group_size=-1)
    codes, scale = torch.zeros(3, 128, dtype=torch.uint8), torch.zeros(3, 1, dtype=torch.float16)
    with pytest.raises(RuntimeError):
        lin(codes, scale, torch.zeros(1, 1, dtype=torch.float16))
    assert not fake.calls
    for zero in (torch.zeros(3, 1), torch.zeros(1, 3, 1), torch.zeros(3, 2)[:, :1]):
        assert lin(codes, scale, zero.half()).shape == (3, 128)
    assert len(fake.calls) == 3


def test_auto_does_without_scratch_that_cannot_be_had(binding, monkeypatch):
    fake = FakeLibrary(4096)
    C = binding(fake)
    args, real = _operands(100), torch.empty

    def empty(*a, dtype=None, **kw):
        if dtype is torch.uint8:
            raise torch.OutOfMemoryError("no memory")
        return real(*a, dtype=dtype, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    C.gemm_i4_dequant(*args)
    assert fake.calls == [(0, None, 0)]
    with pytest.raises(torch.OutOfMemoryError):
        C.gemm_i4_dequant(*args, algo=C.GEMM_GROUP_F8)


def test_recorded_decode_call_keeps_off_the_shared_workspace(binding, monkeypatch):
    counters = []
    fake = FakeLibrary(16384, lambda: counters.append(bytes((ctypes.c_uint8 * 4096).from_address(fake.calls[-1][1]))))
    C = binding(fake)
    monkeypatch.setattr(C, "_WORKSPACES", {})
    args = _operands(16)
    for capturing in (True, False, True):
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
        C.gemm_i4_dequant(*args)
        assert len(C._WORKSPACES) == (len(counters) > 1)            # a recorded call leaves nothing for the others
    (shared,) = C._WORKSPACES.values()
    assert fake.calls[1][1] == shared.data_ptr() != fake.calls[2][1] and not any(map(any, counters))


@pytest.mark.gpu
@pytest.mark.parametrize("warm", [True, False])
def test_recorded_decode_call_outlives_a_larger_call(cuda, warm):
    """The larger call replaces the stream's workspace; other tensors get its memory; the recorded call must not care."""
    m = 64
    t = [_dev(x) for x in make_case(31, m, 12288, 4096, 128, 128, False)[:4]]
    large = [_dev(x) for x in make_case(32, m, 57344, 8192, 128, 128, False)[:4]]
    want, want_large = cuda.gemm_i4_dequant(*t), cuda.gemm_i4_dequant(*large)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        if warm:
            cuda.gemm_i4_dequant(*t)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            d = cuda.gemm_i4_dequant(*t)
        assert torch.equal(cuda.gemm_i4_dequant(*large), want_large)
        junk = [torch.full((10 << 20,), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
        for _ in range(2):
            d.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(d, want)
    assert all(bool((j == 255).all()) for j in junk)


@pytest.mark.gpu
@pytest.mark.parametrize("groups,m,n", [((128, 128, False), 300, 512), ((0, 0, True), 1536, 256)])
def test_two_threads_on_one_stream(cuda, groups, m, n):
    """Different operands from two threads on the default stream: every result is that of its own operands."""
    k, wrong = 2048, []
    work = []
    for seed in (1, 2):
        ap, bp, sa, sb, za, _ = make_case(seed, m, n, k, *groups)
        A, B, SA, SB = (_dev(t) for t in (ap, bp, sa, sb))
        kw = {} if za is None else {"A_zero": _dev(za), "B_rowsum": cuda.weight_rowsum(B, k)}
        work.append(((A, B, SA, SB), kw, _dev(O.gemm_i4_dequant(ap, bp, sa, sb, a_zero=za).view(np.int16))))

    def loop(args, kw, want):
        got = [cuda.gemm_i4_dequant(*args, **kw) for _ in range(200)]
        wrong.append(sum(not torch.equal(d.view(torch.int16), want) for d in got))
    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0]


def _auto(cuda, t, workspace, nbytes):
    m, n, k = t[0].shape[0], t[1].shape[0], 2 * t[0].shape[1]
    d = torch.empty(m, n, dtype=torch.float16, device="cuda")
    rc = cuda._lib.load().flh_b200_gemm_i4_dequant(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), None, t[3].data_ptr(), None, None, d.data_ptr(), m, n, k,
                                                   k // t[2].shape[1], k // t[3].shape[1], 0, 0, workspace, nbytes, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return d


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (16, 4096, 11008), (31, 4096, 4096)])
def test_auto_without_workspace_is_the_single_chain(cuda, m, n, k):
    """Whoever passes no workspace, the reference's own symbol among them, gets the chain of the oracle bit for bit; with the
    workspace of the kernels that split the chain AUTO may take the ring kernel."""
    case = make_case(m + n, m, n, k, 128, 128, False)
    t, want = [_dev(x) for x in case[:4]], _dev(O.gemm_i4_dequant(*case[:4]).view(np.int16))
    lib, ring = cuda._lib.load(), cuda.gemm_i4_dequant(*t, algo=cuda.GEMM_DECODE_RING)
    need = lib.flh_b200_gemm_workspace_bytes(m, n, k, 128, 128, 0)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    assert torch.equal(_auto(cuda, t, None, 0).view(torch.int16), want)
    assert torch.equal(_auto(cuda, t, ws.data_ptr(), need), ring) and torch.equal(cuda.gemm_i4_dequant(*t), ring)
    d = torch.empty(m, n, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    lib.flhDenseLayerGEMM_i4_o16(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), d.data_ptr(), m, n, k)
    torch.cuda.synchronize()
    assert torch.equal(d.view(torch.int16), want)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [16, 64])
def test_scales_off_a_word_boundary_keep_the_workspace(cuda, m):
    """The ring kernel reads group scales as words; others go to the kernel that pick_algo names, with its workspace."""
    t = [_dev(x) for x in make_case(9, m, 4096, 4096, 128, 128, False)[:4]]
    named = cuda._lib.load().flh_b200_gemm_pick_algo(m, 4096, 4096, 128, 128)
    assert torch.equal(cuda.gemm_i4_dequant(*t[:2], _off(t[2], 1), _off(t[3], 1)), cuda.gemm_i4_dequant(*t, algo=named))
    u = [_dev(x) for x in make_case(9, m, 4096, 4096, 0, 0, False)[:4]]
    assert torch.equal(cuda.gemm_i4_dequant(*u[:2], _off(u[2], 1), _off(u[3], 1)), cuda.gemm_i4_dequant(*u, algo=named))
