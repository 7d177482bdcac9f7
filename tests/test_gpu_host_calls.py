"""The native form of the quantiser and linear calls (csrc/host_calls.cpp) against the way in Python: the same bits where it takes
the arguments, the same results and errors where it leaves them to Python."""
import threading
import time

import pytest
import torch

from flh_b200.nn import ActQuantizer, LinearFLH

pytestmark = pytest.mark.gpu


def _both(monkeypatch, cuda, call):
    """call() with the native form and without; what came out (or the error) of each."""
    def one():
        try:
            out = call()
        except (RuntimeError, IndexError, AttributeError, ValueError) as e:
            return type(e), str(e)
        return [t if t is None else (tuple(t.shape), t.dtype, t.stride(), t.cpu()) for t in (out if isinstance(out, tuple) else (out,))]
    assert cuda._host is not None, "build it with python -m flh_b200.build"
    native = one()
    with monkeypatch.context() as m:
        m.setattr(cuda, "_host", None)
        plain = one()
    return native, plain


@pytest.mark.parametrize("shape", [(1, 1, 8), (2, 3, 4096), (5, 257, 1032)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_squares_and_final_norm(cuda, monkeypatch, shape, dtype):
    from flh_b200.model import RMSNorm
    x = (torch.randn(shape, device="cuda") * 8).to(dtype)
    x.view(-1)[:4] = torch.tensor([0.0, -0.0, float("inf"), 6e-8], dtype=dtype)
    assert torch.equal(cuda.square_f32(x), x.float().pow(2))
    norm = RMSNorm(shape[-1], 1e-5).cuda()
    x = x.nan_to_num(posinf=1.0)
    assert torch.equal(norm(x, last=True), norm(x)[:, -1:])
    grad = x.clone().requires_grad_()                    # a derivative has to pass through
    assert cuda.square_f32(grad) is None and norm(grad, last=True).requires_grad
    assert cuda.square_f32(x[..., 1:]) is None and cuda.square_f32(x.float()) is None and cuda.square_f32(x.cpu()) is None


def _same(a, b):
    if isinstance(a, tuple) or isinstance(b, tuple):                      # errors
        return a == b
    return len(a) == len(b) and all((x is None and y is None) or (x[:3] == y[:3] and torch.equal(x[3], y[3])) for x, y in zip(a, b))


def _inputs(k, dtype):
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(6, k, device="cuda", generator=g).to(dtype)
    yield x
    yield x[0]                                                            # one dimension
    yield x.view(2, 3, k)
    yield x[:0]                                                           # no rows
    yield x.t().contiguous().t()                                          # transposed storage
    yield x[:, : k // 2]                                                  # row stride
    yield x.flatten()[1:1 + 5 * k].view(5, k)                             # two bytes off
    yield x.cpu()
    yield x.float()
    yield torch.nn.Parameter(x, requires_grad=False)


@pytest.mark.parametrize("k", [64, 1024, 11008])
@pytest.mark.parametrize("sym,group,had,dtype", [(True, 128, False, torch.float16), (True, 128, True, torch.float16), (True, 32, True, torch.bfloat16),
                                                 (False, -1, False, torch.float16), (False, -1, True, torch.bfloat16)])
def test_quantiser_native_equals_python(cuda, monkeypatch, k, sym, group, had, dtype):
    quant = ActQuantizer(bits=4, group_size=group, sym=sym, use_hadamard=had, packed_output=True)
    for x in _inputs(k, dtype):
        native, plain = _both(monkeypatch, cuda, lambda: quant(x))
        assert _same(native, plain), (tuple(x.shape), x.dtype, x.device, native, plain)


@pytest.mark.parametrize("gs", [32, 64, 128])
def test_scales_of_the_normalised_transform(cuda, monkeypatch, gs):
    """Every size a scale can have: the factor inside the kernel rounds as torch's division behind it."""
    x = torch.zeros(65536, gs, dtype=torch.float16, device="cuda")
    x[:, 0] = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.float16)     # an impulse: all group values are it
    quant = ActQuantizer(bits=4, group_size=gs, sym=True, use_hadamard=True, packed_output=True)
    parts = [x, *x.split(2048)]                          # the kernel of many groups; the kernel of few, which the same values reach in parts
    seen = set()
    for part in parts:
        (s, _, q), (s2, _, q2) = quant(part), (monkeypatch.setattr(cuda, "_host", None), quant(part))[1]
        monkeypatch.undo()
        assert torch.equal(s.view(torch.int16), s2.view(torch.int16)) and torch.equal(q, q2)
        if part is not x:
            seen.update(s.view(torch.int16).unique().tolist())
    assert len(seen) > 10000                             # most are no floor


@pytest.mark.parametrize("m", [1, 16, 64, 130])
@pytest.mark.parametrize("group,zero,bias,out", [(128, False, False, None), (128, False, True, torch.bfloat16), (-1, True, True, None), (-1, False, False, torch.bfloat16)])
def test_linear_native_equals_python(cuda, monkeypatch, m, group, zero, bias, out):
    k, n = 1024, 512
    g = torch.Generator(device="cuda").manual_seed(m)
    lin = LinearFLH(k, n, bias=bias, dtype=torch.float16, device="cuda", group_size=group)
    lin.w_packed.copy_(torch.randint(0, 256, lin.w_packed.shape, dtype=torch.uint8, device="cuda", generator=g))
    lin.w_scale.copy_(torch.rand(lin.w_scale.shape, device="cuda", generator=g) * 0.015 + 0.005)
    if bias:
        lin.bias.copy_(torch.randn(n, device="cuda", generator=g))
    x = torch.randint(0, 256, (m, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    gs = k // 128 if group == 128 else 1
    s = (torch.rand(m, gs, device="cuda", generator=g) + 0.5).half()
    z = torch.randint(0, 16, (m, gs), device="cuda", generator=g).half() if zero else None
    zs = None if z is None else z.view(1, m, gs)
    forms = [(x, s, z), (x.view(1, m, -1), s.view(1, m, gs), zs), (x[:0], s[:0], None if z is None else z[:0]),
             (x, s.t().contiguous().t(), z)]
    for a, b, c in forms:
        native, plain = _both(monkeypatch, cuda, lambda: lin(a, b, c, out_dtype=out))
        assert _same(native, plain), (tuple(a.shape), a.device, native, plain)
    graph = torch.cuda.CUDAGraph()                                       # recorded and replayed
    want = lin(x, s, z, out_dtype=out)
    with torch.cuda.graph(graph):
        y = lin(x, s, z, out_dtype=out)
    y.zero_()
    graph.replay()
    assert torch.equal(y, want)


@pytest.mark.parametrize("what", ["group", "token", "linear", "squares"])
def test_other_threads_run_while_a_call_waits_for_the_queue(cuda, what):
    """Calls behind a kernel of half a second fill the stream's queue (1,024 launches), and the next one waits until that kernel is
    done: meanwhile another thread keeps running.  Its longest pause is bounded by half of the whole time; the interpreter's lock held
    through the wait makes it nearly all of that (what else pauses it is a few switch intervals of 5 ms)."""
    k = 1024
    x = torch.randn(1, 1, k, device="cuda").half()
    packed = torch.randint(0, 256, (1, k // 2), dtype=torch.uint8, device="cuda")
    scale = torch.ones(1, 1, device="cuda", dtype=torch.float16)
    lin = LinearFLH(k, 128, dtype=torch.float16, device="cuda", group_size=-1)
    group = ActQuantizer(bits=4, group_size=128, sym=True, use_hadamard=False, packed_output=True)
    token = ActQuantizer(bits=4, group_size=-1, sym=False, use_hadamard=False, packed_output=True)
    call = {"group": lambda: group(x), "token": lambda: token(x), "linear": lambda: lin(packed, scale), "squares": lambda: cuda.square_f32(x)}[what]
    call()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    ticks, stop = [time.perf_counter()], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    other = threading.Thread(target=tick)
    other.start()
    try:
        start = time.perf_counter()
        torch.cuda._sleep(1_000_000_000)             # clocks
        for _ in range(4000):
            call()
        torch.cuda.synchronize()
        end = time.perf_counter()
    finally:
        stop.set()
        other.join()
    ticks.append(end)
    pause = max(t1 - t0 for t0, t1 in zip(ticks, ticks[1:]))
    assert end - start > 0.3
    assert pause < 0.5 * (end - start), (pause, end - start)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_final_norm_compiled_traced_and_transformed(cuda, dtype):
    """What has to see the operations of the last position's norm sees them: the results are those of the whole norm."""
    from flh_b200.model import RMSNorm

    class Last(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.norm = RMSNorm(256, 1e-5).cuda()

        def forward(self, x):
            return self.norm(x, last=True)

    norm, (x, t) = Last(), torch.randn(2, 2, 3, 256, device="cuda").to(dtype)
    want = norm.norm(x)[:, -1:]
    torch._dynamo.reset()
    assert torch.equal(torch.compile(norm, fullgraph=True, backend="eager")(x), want)
    assert torch.equal(torch.export.export(norm, (x,), strict=True).module()(x), want)
    assert torch.equal(torch.jit.trace(norm, (t,), check_trace=False)(x), want)
    assert torch.equal(torch.vmap(norm)(x[None])[0], want)
    y, dy = torch.func.jvp(norm, (x,), (t,))
    dw = torch.func.jvp(norm.norm, (x,), (t,))[1][:, -1:]
    assert torch.equal(y, want) and torch.equal(dy, dw) and bool(dy.any())
