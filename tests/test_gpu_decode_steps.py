"""The tensor-core decode GEMM where its stages hold two K-blocks (more than 32 tokens, group scales, K a multiple of 256) and beside
that: one step, ranges that end inside a tile, an odd number of K-blocks."""
import pytest
import torch

from oracle import oracle as O
from test_gpu_gemm import DECODE_TC, _close, _dev, make_case, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(33, 128, 256), (64, 256, 512), (50, 384, 896), (64, 1280, 8192), (48, 19200, 1024)])
@pytest.mark.parametrize("mode", [(128, 128, False), (128, 0, False), (0, 128, False), (128, 128, True)])
def test_decode_tc_steps_of_two_blocks(cuda, m, n, k, mode):
    case = make_case(m + n + k, m, n, k, *mode, bias=m == 50)
    if k <= 512:                                         # four K-blocks at least to a CTA: a tile is one chain, bit for bit
        run_case(cuda, DECODE_TC, case)
        return
    ap, bp, sa, sb, za, bi = case
    kw = dict(A_zero=None if za is None else _dev(za), B_rowsum=None if za is None else cuda.weight_rowsum(_dev(bp), 128),
              bias=None if bi is None else _dev(bi), algo=DECODE_TC)
    args = [_dev(t) for t in (ap, bp, sa, sb)]
    d1, d2 = cuda.gemm_i4_dequant(*args, **kw), cuda.gemm_i4_dequant(*args, **kw)
    assert torch.equal(d1.view(torch.int16), d2.view(torch.int16))
    ok, worst = _close(d1, O.gemm_i4_dequant(ap, bp, sa, sb, a_zero=za, bias=bi))     # chains of the CTAs of a tile, added in K order
    assert ok, worst
    torch.cuda.synchronize()
    assert cuda.gemm_status()[0] == 0


@pytest.mark.parametrize("m", [9, 16, 24, 32, 40, 64])
@pytest.mark.parametrize("mode", [(128, 128, False), (128, 128, True), (0, 0, False), (0, 0, True)])
def test_decode_tc_long_ranges(cuda, m, mode):
    """28 K-blocks to a CTA (55 above 32 tokens): every ring of every form goes round several times.  The first and the last 384 channels (whole
    tiles and shared ones) against the oracle."""
    n, k = 16384, 8192
    ap, bp, sa, sb, za, _ = make_case(m, m, n, k, *mode)
    kw = dict(A_zero=None if za is None else _dev(za), B_rowsum=None if za is None else cuda.weight_rowsum(_dev(bp), mode[0] or k), algo=DECODE_TC)
    d = cuda.gemm_i4_dequant(_dev(ap), _dev(bp), _dev(sa), _dev(sb), **kw)
    for part in (slice(0, 384), slice(n - 384, n)):
        want = O.gemm_i4_dequant(ap, bp[part], sa, sb[part], a_zero=za)
        got = d[:, part].contiguous()
        if mode[0] == 0:                                 # int32 sums: the split changes no bit
            assert (got.cpu().numpy().view("u2") == want.view("u2")).all()
        else:
            ok, worst = _close(got, want)
            assert ok, worst
    torch.cuda.synchronize()
    assert cuda.gemm_status()[0] == 0
