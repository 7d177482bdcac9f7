"""GPU parity of the fp8 group-scale GEMM and of the ring decode GEMM against the CPU oracle, at the edges of their tiles."""
import numpy as np
import pytest
import torch

from helpers import rs
from oracle import oracle as O
from test_gpu_gemm import _dev, make_case, run_case

pytestmark = pytest.mark.gpu
F8, RING, AUTO = 9, 11, 0


@pytest.fixture(autouse=True)
def _status_clean(cuda):
    yield
    torch.cuda.synchronize()
    st = cuda.gemm_status()
    assert st[0] == 0, f"a bounded wait ran out: code {st[0]} in CTA {st[1]}"


# one row, both sides of a 256-row tile, a ragged last tile; one K-group, more groups than scale slots, a count that is no
# multiple of eight; more tiles than resident pairs; every scale layout
@pytest.mark.parametrize("m,n,k", [(1, 256, 128), (255, 256, 256), (257, 512, 1024), (515, 1280, 1408), (300, 19200, 256), (700, 768, 11008)])
@pytest.mark.parametrize("mode", [(128, 128, False), (128, 0, False), (0, 128, False)])
def test_group_f8_is_bit_exact(cuda, m, n, k, mode):
    run_case(cuda, F8, make_case(m + n + k, m, n, k, *mode, bias=m == 257), bf16=m == 515)


@pytest.mark.parametrize("a,b", [(0x88, 0x88), (0x88, 0x77), (0x77, 0x77)])
def test_group_f8_extreme_codes(cuda, a, b):
    """Every code at an end of its range: the largest group sums (8192 units), exact in the fp8 tensor core's accumulator."""
    ap, bp, sa, sb, _, _ = make_case(7, 300, 512, 1024, 128, 128, False, neg_scales=True)
    ap[:], bp[:] = a, b
    run_case(cuda, F8, (ap, bp, sa, sb, None, None))


def test_group_f8_needs_its_workspace_and_auto_does_without(cuda):
    lib, m, n, k = cuda._lib.load(), 300, 512, 2048
    case = make_case(11, m, n, k, 128, 128, False)
    run_case(cuda, AUTO, case)
    A, B, SA, SB = (_dev(t) for t in case[:4])
    D = torch.empty(m, n, dtype=torch.float16, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    call = lambda algo, ws, nbytes: lib.flh_b200_gemm_i4_dequant(A.data_ptr(), B.data_ptr(), SA.data_ptr(), None, SB.data_ptr(), None, None, D.data_ptr(),
                                                                 m, n, k, 128, 128, 0, algo, ws, nbytes, s)
    need = lib.flh_b200_gemm_workspace_bytes(m, n, k, 128, 128, F8)
    assert need == lib.flh_b200_gemm_workspace_bytes(m, n, k, 128, 128, cuda.GEMM_AUTO_WORKSPACE)      # AUTO would take it
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    assert call(F8, None, 0) != 0 and call(F8, ws.data_ptr(), need - 1) != 0
    want = O.gemm_i4_dequant(*case[:4]).view(np.uint16)
    for w, nbytes in ((None, 0), (ws.data_ptr(), need - 1), (ws.data_ptr(), need)):
        D.zero_()
        assert call(AUTO, w, nbytes) == 0
        assert np.array_equal(D.cpu().numpy().view(np.uint16), want)


def test_group_f8_scratch_of_a_captured_call_outlives_a_larger_call(cuda):
    """A recorded launch keeps its own scratch: a later, larger call on the same stream must not take it away."""
    small, large = make_case(21, 300, 512, 2048, 128, 128, False), make_case(22, 600, 1024, 4096, 128, 128, False)
    t = [_dev(x) for x in small[:4]]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        cuda.gemm_i4_dequant(*t)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            d = cuda.gemm_i4_dequant(*t)
        run_case(cuda, AUTO, large)
        junk = [torch.full((4 << 20,), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
        g.replay()
        torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint16), O.gemm_i4_dequant(*small[:4]).view(np.uint16))
    del junk


SHAPES = [(128, 128), (64 * 3 * 2, 1152), (256, 2048), (512, 11008), (19200, 384)]   # half a chunk, half a stage, one stage, many; many tiles


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("asym", [False, True])
def test_ring_without_group_scales_is_bit_exact(cuda, m, n, k, asym):
    run_case(cuda, RING, make_case(m + n + k, m, n, k, 0, 0, asym, bias=m == 9), bf16=m == 17)


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("mode", [(128, 128, False), (128, 0, False), (0, 128, False)])
def test_ring_with_group_scales(cuda, m, n, k, mode):
    """A warp keeps the binary32 chain of its K-groups and the chains are added: each order of G terms is within
    G 2^-24 sum |terms| of the exact sum, so two orders differ by at most twice that, and the result by one ulp (2^-10) of its
    own rounding on top.  The same bits on every run."""
    ap, bp, sa, sb, _, _ = make_case(m + n + k, m, n, k, *mode)
    args = [_dev(t) for t in (ap, bp, sa, sb)]
    d1, d2 = cuda.gemm_i4_dequant(*args, algo=RING), cuda.gemm_i4_dequant(*args, algo=RING)
    assert torch.equal(d1.view(torch.int16), d2.view(torch.int16))
    G = k // 128
    a = np.abs(O.unpack_i4(ap).astype(np.float64)).reshape(m, G, 128) * np.broadcast_to(sa.astype(np.float64), (m, G))[:, :, None]
    b = np.abs(O.unpack_i4(bp).astype(np.float64)).reshape(n, G, 128) * np.broadcast_to(sb.astype(np.float64), (n, G))[:, :, None]
    bound = 2 * G * 2.0 ** -24 * (a.reshape(m, k) @ b.reshape(n, k).T)
    ref = O.gemm_i4_dequant(ap, bp, sa, sb).astype(np.float64)
    err = np.abs(d1.cpu().numpy().astype(np.float64) - ref)
    assert (err <= bound + 2.0 ** -10 * np.abs(ref) + 2.0 ** -24).all(), err.max()


@pytest.mark.parametrize("bf16", [False, True])
def test_silu_of_every_gate(cuda, bf16):
    """SiLU rounds a function of one 16-bit value: all 65,536 of them (but NaN), beside two values of up."""
    bits = np.arange(65536, dtype=np.uint16)
    g = O.bf16_bits_to_f32(bits) if bf16 else bits.view(np.float16).astype(np.float32)
    bits = bits[~np.isnan(g)]
    bits = np.concatenate([bits, bits[:(-len(bits)) % 64]])
    up = (O.f32_to_bf16_bits(np.array([1.0, -2.75], np.float32)) if bf16 else np.array([1.0, -2.75], np.float16)).view(np.uint16)
    gu = np.stack([np.concatenate([bits, np.full_like(bits, u)]) for u in up])
    x = torch.from_numpy(gu.view(np.int16)).cuda().view(torch.bfloat16 if bf16 else torch.float16)
    want = O.silu_mul16(gu if bf16 else gu.view(np.float16), bf16=bf16)
    got = cuda.silu_mul(x).view(torch.int16).cpu().numpy().view(np.uint16)
    assert np.array_equal(got, want.view(np.uint16))


@pytest.mark.parametrize("bf16", [False, True])
def test_silu_of_every_gate_among_ordinary_ones(cuda, bf16):
    """A group of eight takes the packed form unless one of its gates is out of that form's range: every 16-bit gate, NaN
    included, in a group whose other seven are ordinary, so that each value meets the form that data sends it to; up runs
    over ordinary, tiny, huge, zero, infinite and NaN values.  All results bit for bit (any NaN for a NaN)."""
    f32 = (lambda b: O.bf16_bits_to_f32(b)) if bf16 else (lambda b: b.view(np.float16).astype(np.float32))
    n = 65536
    gate = rs(8).standard_normal((n, 8)).astype(np.float32) * 3.0
    gate = O.f32_to_bf16_bits(gate) if bf16 else gate.astype(np.float16).view(np.uint16)
    gate[np.arange(n), rs(9).randint(0, 8, n)] = rs(10).permutation(n).astype(np.uint16)
    gate = gate.reshape(64, -1)
    with np.errstate(over="ignore", invalid="ignore"):
        special = np.array([1.0, -2.75, 1e-7, -1e-30, 6e4, 3e38, 0.0, -0.0, np.inf, np.nan], np.float32)
        special = O.f32_to_bf16_bits(special) if bf16 else special.astype(np.float16).view(np.uint16)
        up = special[rs(11).randint(0, 10, gate.shape)]
        gu = np.concatenate([gate, up], axis=1)
        want = O.silu_mul16(gu if bf16 else gu.view(np.float16), bf16=bf16).view(np.uint16)
    x = torch.from_numpy(gu.view(np.int16)).cuda().view(torch.bfloat16 if bf16 else torch.float16)
    got = cuda.silu_mul(x).view(torch.int16).cpu().numpy().view(np.uint16)
    nan = np.isnan(f32(want))
    assert np.array_equal(np.isnan(f32(got)), nan)
    bad = (got != want) & ~nan
    assert not bad.any(), [(hex(g), hex(u), hex(a), hex(b)) for g, u, a, b in zip(gate[bad][:8], up[bad][:8], got[bad][:8], want[bad][:8])]


@pytest.mark.parametrize("D,B,S", [(128, 2, 40), (128, 3, 1), (40, 1, 700), (8, 2, 3)])
def test_rope_by_token_is_the_transposed_form(cuda, D, B, S):
    nh, nkv, cur, T = 6, 2, 3, S + 5
    g = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randn(B * S, (nh + 2 * nkv) * D, device="cuda", generator=g).half()
    ang = torch.randn(S, D // 2, device="cuda", generator=g)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    outs = []
    for by_token in (False, True):
        kc, vc = torch.zeros(B, nkv, T, D, device="cuda").half(), torch.zeros(B, nkv, T, D, device="cuda").half()
        q = torch.empty((B, S, nh, D) if by_token else (B, nh, S, D), dtype=torch.float16, device="cuda")
        cuda.rope_kv(qkv, cos, sin, q, kc, vc, B, S, nh, nkv, cur, q_by_token=by_token)
        outs.append((q.transpose(1, 2) if by_token else q, kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    x = qkv.view(B, S, nh + 2 * nkv, D)[:, :, :nh].float()
    c, s = cos[None, :, None], sin[None, :, None]
    want = torch.cat((x[..., :D // 2] * c - x[..., D // 2:] * s, x[..., D // 2:] * c + x[..., :D // 2] * s), -1).half()
    assert torch.equal(outs[0][0], want.transpose(1, 2))


@pytest.mark.parametrize("m,k", [(1, 8), (3, 2056), (16, 4096), (33, 8192)])
def test_rmsnorm(cuda, m, k):
    """Against 64 bits: one ulp of each of the two float16 roundings (2^-10 each), the binary32 part far below that."""
    from flh_b200.model import RMSNorm
    x = torch.from_numpy(rs(m + k).standard_normal((m, k + 8)).astype(np.float16)).cuda()[:, :k]
    norm = RMSNorm(k, 1e-5).cuda()
    norm.weight.data.copy_(torch.from_numpy(rs(5).uniform(0.5, 2.0, k).astype(np.float16)))
    v = x.double()
    want = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5) * norm.weight.double()
    err = (norm(x).double() - want).abs()
    assert bool((err <= 2.0 ** -9 * want.abs() + 2.0 ** -24).all()), err.max().item()


def _norm_of(k):
    from flh_b200.model import RMSNorm
    norm = RMSNorm(k, 1e-5).cuda()
    norm.weight.data.copy_(torch.from_numpy(rs(5).uniform(0.5, 2.0, k).astype(np.float16)))
    return norm, lambda x: (x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5)).to(x.dtype) * norm.weight


@pytest.mark.parametrize("m,k", [(1, 8), (1, 4096), (3, 2056), (16, 4096), (700, 4096), (33, 8192)])
@pytest.mark.parametrize("layout", ["contiguous", "strided", "misaligned"])
def test_rmsnorm_has_the_bits_of_the_tensor_operations(cuda, m, k, layout):
    norm, want = _norm_of(k)
    x = torch.from_numpy(rs(m + k).standard_normal(m * (k + 8) + 1).astype(np.float16)).cuda()
    x = {"contiguous": x[:m * k].view(m, k), "strided": x[:-1].view(m, k + 8)[:, :k], "misaligned": x[1:1 + m * k].view(m, k)}[layout]
    assert torch.equal(norm(x).view(torch.int16), want(x).view(torch.int16))


def test_rmsnorm_under_tangents_vmap_and_tracing(cuda):
    norm, want = _norm_of(256)
    x, t = (torch.from_numpy(rs(s).standard_normal((4, 256)).astype(np.float16)).cuda() for s in (1, 2))
    y, dy = torch.func.jvp(norm, (x,), (t,))
    assert torch.equal(y, want(x)) and torch.equal(dy, torch.func.jvp(want, (x,), (t,))[1]) and bool(dy.any())
    assert torch.equal(torch.vmap(norm)(x), torch.vmap(want)(x))
    traced = torch.jit.trace(norm, (x,), check_trace=False)
    assert torch.equal(traced(t), want(t))


def test_rmsnorm_refuses_another_width(cuda):
    norm, _ = _norm_of(256)
    for k in (128, 512):
        with pytest.raises(RuntimeError):
            norm(torch.zeros(2, k, dtype=torch.float16, device="cuda"))


@pytest.mark.parametrize("shape", [(128,), (3, 256), (2, 5, 384)])
@pytest.mark.parametrize("kind", ["group", "group_had", "token"])
def test_quantiser_module_shapes_and_strides(cuda, shape, kind):
    """The module's outputs follow the input's leading dimensions, contiguous or not, as the functions on matrices give them."""
    from flh_b200.nn import ActQuantizer
    sym, had = kind != "token", kind == "group_had"
    quant = ActQuantizer(bits=4, group_size=128 if sym else -1, sym=sym, use_hadamard=had, packed_output=True)
    K = shape[-1]
    base = torch.randn(shape[:-1] + (K + 64,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).half()
    for x in (base[..., :K].contiguous(), base[..., :K]):
        s, z, q = quant(x)
        flat = x.reshape(-1, K).contiguous()
        if sym:
            q0, s0 = (cuda.hadamard_and_quantize_i4 if had else cuda.quant_and_pack_i4)(flat.view(-1, 128))
            s0 = s0 / 128 ** 0.5 if had else s0
            assert z is None and s.shape == shape[:-1] + (K // 128,)
        else:
            q0, s0, z0 = cuda.quant_token_asym_i4(flat, hadamard=False)
            assert s.shape == z.shape == shape[:-1] + (1,) and torch.equal(z.reshape(-1), z0)
        assert q.shape == shape[:-1] + (K // 2,) and torch.equal(q.reshape(-1), q0.reshape(-1)) and torch.equal(s.reshape(-1), s0.reshape(-1))
    with pytest.raises(RuntimeError):
        ActQuantizer(bits=4, group_size=128, sym=True, use_hadamard=False, packed_output=True)(torch.zeros(2, 192, device="cuda").half())


@pytest.mark.parametrize("kind", ["group", "group_had", "token"])
@pytest.mark.parametrize("shape", [(0, 64), (2, 0, 256)])
def test_quantiser_module_on_no_rows(cuda, kind, shape):
    from flh_b200.nn import ActQuantizer
    sym = kind != "token"
    quant = ActQuantizer(bits=4, group_size=128 if sym else -1, sym=sym, use_hadamard=kind == "group_had", packed_output=True)
    s, z, q = quant(torch.empty(shape, dtype=torch.float16, device="cuda"))
    assert q.shape == shape[:-1] + (shape[-1] // 2,) and s.shape == shape[:-1] + (shape[-1] // 128 if sym else 1,) and (z is None) == sym
