"""The prompt products QMatMul.forward runs: f16 operands holding integers, weights expanded into tensor memory.

Q4_K / Q6_K (cq_prompt_matmul) against the CPU path's matmul (the tolerance of the other prompt tests: only the order of f32
additions differs), and bit for bit against the int8 kernel behind cq_prefill_gemm: the same integers, the same f32 operations
in the same order.
"""
import numpy as np
import pytest
import torch

from candle_b200 import capi
from candle_b200.quantized import GgmlDType, QMatMul, QTensor
from helpers import TSIZE, make_case, rel_err

pytestmark = pytest.mark.gpu
ELEM = {torch.float32: capi.F32, torch.float16: capi.F16, torch.bfloat16: capi.BF16}


def _run(scratch_bytes, matmul, flag, wtype, w_dev, x_dev, k, n):
    tokens, st = x_dev.shape[0], torch.cuda.current_stream().cuda_stream
    scratch = torch.full((scratch_bytes + 64,), 0xFF, dtype=torch.uint8, device=x_dev.device)     # 0xFFFF: f16 NaN
    out = torch.full((tokens * n + 32,), float("nan"), dtype=x_dev.dtype, device=x_dev.device)
    matmul(wtype, w_dev.data_ptr(), x_dev.data_ptr(), ELEM[x_dev.dtype], out.data_ptr(), scratch.data_ptr(), k, n, tokens, n, st)
    capi.check("prompt")
    torch.cuda.synchronize()
    assert flag() == 0
    assert bool((scratch[-64:] == 0xFF).all()), "scratch written past its end"
    assert bool(torch.isnan(out[tokens * n:].float()).all()) and not bool(torch.isnan(out[:tokens * n].float()).any())
    return out[:tokens * n].view(tokens, n)


def _prompt(lib, wtype, w_dev, x_dev, k, n):
    return _run(lib.cq_prompt_scratch_bytes(x_dev.shape[0], k), lib.cq_prompt_matmul, lib.cq_prompt_timeout_flag, wtype, w_dev, x_dev, k, n)


def _int8(lib, wtype, w_dev, x_dev, k, n):
    tokens, st = x_dev.shape[0], torch.cuda.current_stream().cuda_stream
    scratch = torch.zeros(lib.cq_prefill_scratch_bytes(tokens, k), dtype=torch.uint8, device=x_dev.device)
    out = torch.empty((tokens, n), dtype=x_dev.dtype, device=x_dev.device)
    lib.cq_prefill_quantize(x_dev.data_ptr(), ELEM[x_dev.dtype], scratch.data_ptr(), k, tokens, st)
    lib.cq_prefill_gemm(wtype, w_dev.data_ptr(), scratch.data_ptr(), out.data_ptr(), ELEM[x_dev.dtype], k, n, tokens, n, st)
    capi.check("prefill")
    return out


# one super-block, one ragged row tile; a full tile and one row more; tokens around the multiples of 16 and of 128; more tiles
# than SMs (several per CTA); K whose Q6_K rows start off a 16-byte boundary (256, 768, 1280) and on one (2048)
@pytest.mark.parametrize("tokens,k,n", [(1, 256, 1), (17, 512, 65), (16, 256, 128), (128, 768, 129), (129, 1280, 200), (333, 2048, 512),
                                        (300, 4096, 96), (2000, 512, 2050)])
@pytest.mark.parametrize("wtype,dtype", [(12, torch.float32), (14, torch.float32), (12, torch.bfloat16), (14, torch.float16)])
def test_prompt_matmul(lib, oracle, cuda_dev, tokens, k, n, wtype, dtype):
    _, x, wq = make_case(oracle, wtype, k, n, tokens, seed=tokens + k + n)
    if wtype == 14:     # negative, zero and extreme sub-block scales
        wq.reshape(-1, 210)[0, 192:208] = np.array([-128, 127, 0, -1, 1, -64, 64, 5, -5, 100, -100, 33, -33, 2, -2, 0], dtype=np.int8).view(np.uint8)
    x_dev = torch.from_numpy(x).to(cuda_dev).to(dtype)
    w_dev = torch.from_numpy(wq).to(cuda_dev)
    out = _prompt(lib, wtype, w_dev, x_dev, k, n)
    if dtype == torch.float32 and tokens <= 333:
        assert rel_err(out.cpu().numpy(), oracle.matmul(wtype, x, wq, n)) <= 1e-5
    assert torch.equal(out, _int8(lib, wtype, w_dev, x_dev, k, n))


def _large_sums(wtype, n, k, kind, rng):
    """Blocks whose integer sums leave 24 bits: scales and codes near their largest, odd ones among them.  "two signs": the second
    half of a super-block takes back what the first has added."""
    nsb = k // 256
    b = rng.integers(0, 256, (n * nsb, TSIZE[wtype]), dtype=np.uint8)
    d = (rng.random((n * nsb, 2)) * 1e-4 + 1e-4).astype(np.float16)
    if wtype == 12:
        b[:, :4] = d.view(np.uint8)
        b[:, 4:16] = 0xFF                                        # scales and minima 63
        b[:, 16:] |= 0 if kind == "two signs" else 0xCC          # codes any, or 12 .. 15
    else:
        b[:, :192] |= 0xFC                                       # codes 60 .. 63
        sc = rng.integers(117, 128, (n * nsb, 16)).astype(np.int8)
        if kind == "two signs":
            sc[:, 8:] *= -1
        b[:, 192:208] = sc.view(np.uint8)
        b[:, 208:] = d[:, :1].view(np.uint8)
    return b.reshape(n, -1)


# every accumulator of a tile: two halves of the tokens, ragged ones, a tile of 16
@pytest.mark.parametrize("tokens", [16, 40, 128, 150])
@pytest.mark.parametrize("wtype", [12, 14])
@pytest.mark.parametrize("kind", ["one sign", "two signs", "some super-blocks"])
def test_prompt_matmul_of_sums_past_24_bits(lib, oracle, cuda_dev, tokens, wtype, kind):
    """The integers are exact for any data (activations of one sign reach +-127 throughout): the bits of the int32 accumulators."""
    rng = np.random.default_rng(tokens + wtype)
    k, n = (1024, 200) if kind != "some super-blocks" else (2304, 20000)        # the second: several tiles per CTA
    wq = _large_sums(wtype, n, k, kind, rng)
    x = (1.0 - 0.06 * rng.random((tokens, k))).astype(np.float32)
    x[1::3] *= -1
    if kind == "some super-blocks":         # 1, 4, 5, 6 of one sign (6 for one token only), the others normal
        other = ~np.isin(np.arange(k) // 256, (1, 4, 5, 6))
        x[:, other] = rng.standard_normal((tokens, int(other.sum())))
        x[:tokens - 1, 6 * 256:7 * 256] = rng.standard_normal((tokens - 1, 256))
    if kind == "two signs" and wtype == 12:
        x[:, np.arange(k) % 256 >= 128] *= -1
    x_dev, w_dev = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev)
    out = _prompt(lib, wtype, w_dev, x_dev, k, n)
    assert torch.equal(out, _int8(lib, wtype, w_dev, x_dev, k, n))
    if kind == "one sign":
        assert rel_err(out.cpu().numpy(), oracle.matmul(wtype, x, wq, n)) <= 1e-5


@pytest.mark.parametrize("wtype", [12, 14])
def test_prompt_matmul_of_non_finite_activations(lib, oracle, cuda_dev, wtype):
    """NaN and infinite activations (int8 -128): the same bits, NaNs in the same places, the other tokens untouched."""
    _, x, wq = make_case(oracle, wtype, 512, 65, 40, seed=9)
    x[3, 5], x[7, ::2], x[11, 300], x[13, 256:] = np.nan, np.nan, np.inf, -np.inf
    x[17] = 1e-41
    x_dev, w_dev = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev)
    scratch, out = torch.zeros(lib.cq_prompt_scratch_bytes(40, 512), dtype=torch.uint8, device=cuda_dev), torch.empty((40, 65), device=cuda_dev)
    lib.cq_prompt_matmul(wtype, w_dev.data_ptr(), x_dev.data_ptr(), capi.F32, out.data_ptr(), scratch.data_ptr(), 512, 65, 40, 65, torch.cuda.current_stream().cuda_stream)
    capi.check("prompt")
    assert torch.equal(out.nan_to_num(1e30, 2e30, 3e30), _int8(lib, wtype, w_dev, x_dev, 512, 65).nan_to_num(1e30, 2e30, 3e30))


def test_prompt_matmul_unaligned_activations(lib, oracle, cuda_dev):
    _, x, wq = make_case(oracle, 12, 512, 70, 40, seed=3)
    w_dev = torch.from_numpy(wq).to(cuda_dev)
    buf = torch.zeros(40 * 512 + 1, device=cuda_dev)
    buf[1:] = torch.from_numpy(x).to(cuda_dev).view(-1)
    assert torch.equal(_prompt(lib, 12, w_dev, buf[1:].view(40, 512), 512, 70), _prompt(lib, 12, w_dev, buf[1:].clone().view(40, 512), 512, 70))


# ---- activation scales per 32 elements ------------------------------------------------------------------------------
NAMES = {2: "Q4_0", 3: "Q4_1", 6: "Q5_0", 7: "Q5_1", 8: "Q8_0", 10: "Q2K", 11: "Q3K", 13: "Q5K"}


def _prompt32(lib, wtype, w_dev, x_dev, k, n):
    return _run(lib.cq_prompt32_scratch_bytes(wtype, x_dev.shape[0], k), lib.cq_prompt32_matmul, lib.cq_prompt32_timeout_flag, wtype, w_dev,
                x_dev, k, n)


@pytest.mark.parametrize("tokens,k,n", [(1, 256, 1), (9, 512, 65), (64, 256, 128), (65, 768, 129), (128, 1280, 200), (200, 2048, 300),
                                        (2000, 512, 2050)])
@pytest.mark.parametrize("wtype", sorted(NAMES))
def test_prompt32_matmul(lib, oracle, cuda_dev, tokens, k, n, wtype):
    _, x, wq = make_case(oracle, wtype, k, n, tokens, seed=tokens + k + n)
    x_dev, w_dev = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev)
    out = _prompt32(lib, wtype, w_dev, x_dev, k, n)
    if wtype in (2, 8):     # the int8 kernel's integers and f32 operations in its order: the same bits
        scratch = torch.zeros(lib.cq_prefill32_scratch_bytes(tokens, k), dtype=torch.uint8, device=cuda_dev)
        ref, st = torch.empty_like(out), torch.cuda.current_stream().cuda_stream
        lib.cq_prefill32_quantize(x_dev.data_ptr(), capi.F32, scratch.data_ptr(), k, tokens, st)
        lib.cq_prefill32_gemm(wtype, w_dev.data_ptr(), scratch.data_ptr(), ref.data_ptr(), capi.F32, k, n, tokens, n, st)
        capi.check("prefill32")
        assert torch.equal(out, ref)
    else:                   # f32 sums in another order
        pick = np.unique(np.linspace(0, tokens - 1, 64).astype(int))
        ref = oracle.cuda_mmvq(wtype, wq, oracle.cuda_quantize_q8_1(x[pick]), k, n)
        assert rel_err(out.cpu().numpy()[pick], ref) <= 2e-6


@pytest.mark.parametrize("wtype", [3, 6, 7])
def test_prompt32_of_block_sums_past_f16(lib, oracle, cuda_dev, wtype):
    """Q8_1's stored sum is infinite where 32 inputs add up to more than 65504: infinities and NaNs where the decode kernel has them."""
    k, n, m = 512, 96, 16
    _, x, wq = make_case(oracle, wtype, k, n, m, seed=1)
    x[3, 64:96], x[5, 32:64], x[5, 300:330], x[7, 480:] = 3000.0, -2500.0, 4000.0, np.nan
    x_dev, w_dev, st = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev), torch.cuda.current_stream().cuda_stream
    y8, decode, out = torch.zeros((m, k // 32, 36), dtype=torch.uint8, device=cuda_dev), torch.empty((m, n), device=cuda_dev), torch.empty((m, n), device=cuda_dev)
    lib.cq_quantize_act(x_dev.data_ptr(), capi.F32, y8.data_ptr(), k, k, m, 0, st)
    for r in range(0, m, 8):
        lib.cq_mmvq(wtype, 0, capi.F32, w_dev.data_ptr(), y8[r:].data_ptr(), decode[r:].data_ptr(), k, n, k // 32, n, 8, st)
    scratch = torch.zeros(lib.cq_prompt32_scratch_bytes(wtype, m, k), dtype=torch.uint8, device=cuda_dev)
    lib.cq_prompt32_matmul(wtype, w_dev.data_ptr(), x_dev.data_ptr(), capi.F32, out.data_ptr(), scratch.data_ptr(), k, n, m, n, st)
    capi.check("prompt32")
    assert torch.equal(torch.isnan(out), torch.isnan(decode)) and torch.equal(torch.isinf(out), torch.isinf(decode))
    assert torch.equal(out[torch.isinf(out)], decode[torch.isinf(decode)]) and not bool(torch.isfinite(out[[3, 5, 7]]).all())
    ok = [i for i in range(m) if i not in (3, 5, 7)]
    assert rel_err(out[ok].cpu().numpy(), decode[ok].cpu().numpy()) <= 2e-6


@pytest.mark.parametrize("wtype", [7, 8, 10, 11, 13])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_prompt32_half_types(lib, oracle, cuda_dev, wtype, dtype):
    """16-bit activations give the f32 result of the same values, rounded once."""
    _, x, wq = make_case(oracle, wtype, 1024, 130, 77, seed=5)
    w_dev, xt = torch.from_numpy(wq).to(cuda_dev), torch.from_numpy(x).to(cuda_dev).to(dtype)
    assert torch.equal(_prompt32(lib, wtype, w_dev, xt, 1024, 130), _prompt32(lib, wtype, w_dev, xt.float(), 1024, 130).to(dtype))


@pytest.mark.parametrize("wtype", [3, 10, 13])
def test_qmatmul_routes_rows_past_one_decode_launch(oracle, cuda_dev, wtype):
    """Rows 9 and up of the Q8_1 formats go to the prompt kernel: the values of the decode kernel, f32 sums in another order."""
    _, x, wq = make_case(oracle, wtype, 512, 96, 21, seed=8)
    mm = QMatMul.from_qtensor(QTensor.from_data(wq, GgmlDType[NAMES[wtype]], (96, 512), cuda_dev))
    xd = torch.from_numpy(x).to(cuda_dev)
    y = mm.forward(xd.view(3, 7, 512)).view(21, 96)
    ref = torch.cat([mm.forward(xd[i:i + 7]) for i in (0, 7, 14)])
    assert rel_err(y.cpu().numpy(), ref.cpu().numpy()) <= 2e-6


@pytest.mark.parametrize("one_sign", [False, True])
@pytest.mark.parametrize("wtype,scale,minimum,mid", [(3, 0, 2, -7.5), (6, 0, None, 0.0), (7, 0, 2, -15.5), (10, 80, 82, 1.5), (11, 108, None, 0.0), (13, 0, 2, 15.5)])
def test_prompt32_is_no_further_from_64_bits_than_the_decode_kernel(lib, cuda_dev, wtype, scale, minimum, mid, one_sign):
    """Weights around zero, whose codes' part and minimum's part nearly cancel in every block.  `scale`, `minimum`: where a block keeps
    its f16 fields; the minimum is `mid` scales, the middle of the codes.  10 % for the two kernels' different roundings."""
    n, m, k = 96, 64, 4096
    per = 32 if wtype < 10 else 256
    gen = torch.Generator(device=cuda_dev).manual_seed(wtype)
    b = torch.randint(0, 256, (n * k // per, TSIZE[wtype]), dtype=torch.uint8, device=cuda_dev, generator=gen)

    def put(b, off, v):
        b[:, off:off + 2] = v.to(torch.float16).view(torch.uint8).view(-1, 2)

    def values(b, d, mn):           # the integers of all elements (d = 1, minimum 0), or the minima's (d = 0, minimum 1), exact in f32
        b = b.clone()
        put(b, scale, torch.full((b.shape[0],), d, device=cuda_dev))
        if minimum is not None:
            put(b, minimum, torch.full((b.shape[0],), mn, device=cuda_dev))
        return QTensor.from_device_blocks(b.reshape(-1), GgmlDType(wtype), (n, k)).dequantize(torch.float32).double()

    d = ((torch.rand(b.shape[0], device=cuda_dev, generator=gen) * 0.5 + 0.75) * 1e-3).half().float()
    put(b, scale, d)
    if minimum is not None:
        put(b, minimum, d * mid)
    if wtype == 10:                 # minima codes = scale codes
        b[:, :16] = (b[:, :16] & 15) * 17
    if wtype == 13:                 # the same in the 6-bit fields
        b[:, 8:12] = b[:, 4:8]
        b[:, 12:16] = (b[:, 12:16] & 15) * 17
    spread = lambda off: b[:, off:off + 2].contiguous().view(torch.float16).double().view(n, -1).repeat_interleave(per, 1)
    codes, dw = values(b, 1.0, 0.0), spread(scale)
    mins = values(b, 0.0, 1.0) * spread(minimum) if minimum is not None else torch.zeros_like(dw)
    if wtype == 6:                  # Q5_0: the kernels take the codes unsigned and -16 d as the minimum
        codes, mins = codes + 16, -16 * dw
    x = torch.randn(m, k, device=cuda_dev, generator=gen)
    x = x.abs() if one_sign else x
    st = torch.cuda.current_stream().cuda_stream
    y8 = torch.zeros((m, k // 32, 36), dtype=torch.uint8, device=cuda_dev)
    lib.cq_quantize_act(x.data_ptr(), capi.F32, y8.data_ptr(), k, k, m, 0, st)
    a = y8.view(-1, 36)
    da = a[:, 0:2].contiguous().view(torch.float16).double().view(m, -1).repeat_interleave(32, 1)
    xq = da * a[:, 4:].contiguous().view(torch.int8).double().view(m, k)
    ref = xq @ (dw * codes).t()
    if wtype in (3, 6, 7):          # the stored f16 sum of a block's inputs
        ref += a[:, 2:4].contiguous().view(torch.float16).double().view(m, -1) @ mins[:, ::32].t()
    else:
        ref += xq @ mins.t()
    wq = b.reshape(n, -1)
    decode = torch.empty((m, n), device=cuda_dev)
    for r in range(0, m, 8):
        lib.cq_mmvq(wtype, 0, capi.F32, wq.data_ptr(), y8[r:].data_ptr(), decode[r:].data_ptr(), k, n, k // 32, n, 8, st)
    capi.check("decode")
    err = lambda o: float((o.double() - ref).norm() / ref.norm())
    assert err(decode) <= 1e-6      # the reference is that arithmetic
    assert err(_prompt32(lib, wtype, wq, x, k, n)) <= 1.1 * err(decode)


MINIMUM = {2: (0, None, 0.0), 8: (0, None, 0.0), 3: (0, 2, -7.5), 6: (0, None, 0.0), 7: (0, 2, -15.5), 10: (80, 82, 1.5), 11: (108, None, 0.0), 13: (0, 2, 15.5)}     # where d and the minimum are; the middle of the codes


def _weights32(wtype, n, k, minimum, gen, dev):
    """Random blocks with minima of `minimum` x the middle of the codes (1: weights around zero; -1: all of one sign, 0: none, 8: the minimum is most of a
    weight), and what they hold, in f64: integers [n, k], scales [n, k / 32] and minima [n, k / 32, 1 or 2]."""
    per, (at_d, at_m, mid) = 32 if wtype < 10 else 256, MINIMUM[wtype]
    b = torch.randint(0, 256, (n * k // per, TSIZE[wtype]), dtype=torch.uint8, device=dev, generator=gen)

    def put(b, off, v):
        b[:, off:off + 2] = v.to(torch.float16).view(torch.uint8).view(-1, 2)

    d = ((torch.rand(b.shape[0], device=dev, generator=gen) * 0.5 + 0.75) * 1e-3).half().float()
    put(b, at_d, d)
    if at_m is not None:
        put(b, at_m, d * mid * minimum)

    def values(d, m):
        c = b.clone()
        put(c, at_d, torch.full((b.shape[0],), d, device=dev))
        if at_m is not None:
            put(c, at_m, torch.full((b.shape[0],), m, device=dev))
        return QTensor.from_device_blocks(c.reshape(-1), GgmlDType(wtype), (n, k)).dequantize(torch.float32).double()

    spread = lambda off: b[:, off:off + 2].contiguous().view(torch.float16).double().view(n, -1).repeat_interleave(per // 32, 1)
    codes, scales = values(1.0, 0.0), spread(at_d)
    if wtype == 6:          # the codes are unsigned, -16 d is the minimum
        return b.reshape(n, -1), codes + 16, scales, -16 * scales.unsqueeze(-1)
    if at_m is None:
        return b.reshape(n, -1), codes, scales, torch.zeros((n, k // 32, 1), dtype=torch.float64, device=dev)
    mins = values(0.0, 1.0)[:, ::16 if wtype == 10 else 32].reshape(n, k // 32, -1)
    return b.reshape(n, -1), codes, scales, mins * spread(at_m).unsqueeze(-1)


def _activations32(lib, wtype, x):
    """What the quantizer makes of them, in f64: integers [m, k], scales [m, k / 32] and sums [m, k / 32, 1 or 2]."""
    m, k = x.shape
    y8 = torch.zeros((m, k // 32, 36), dtype=torch.uint8, device=x.device)
    lib.cq_quantize_act(x.data_ptr(), capi.F32, y8.data_ptr(), k, k, m, 0, torch.cuda.current_stream().cuda_stream)
    a = y8.view(-1, 36)
    d, q = a[:, 0:2].contiguous().view(torch.float16).double().view(m, -1), a[:, 4:].contiguous().view(torch.int8).double().view(m, k)
    if wtype < 10:
        return q, d, a[:, 2:4].contiguous().view(torch.float16).double().view(m, -1, 1)
    return q, d, d.unsqueeze(-1) * q.view(m, k // 32, 2 if wtype == 10 else 1, -1).sum(-1)


def _plain_sums(wtype, codes, scales, mins, q, d, sums):
    """The sums with a minimum added per block, in f32 (operations on f64 values, rounded; products of two f32 are exact in f64): the blocks of 256 elements one
    after the other, the 256s by a two-sum.  Also the exact result."""
    r = lambda v: v.float().double()
    m, n, nb = q.shape[0], codes.shape[0], d.shape[1]
    total, low, acc, exact = (torch.zeros((m, n), dtype=torch.float64, device=q.device) for _ in range(4))
    for b in range(nb):
        i = q[:, 32 * b:32 * b + 32] @ codes[:, 32 * b:32 * b + 32].t()
        dd, dw, terms = d[:, b:b + 1], scales[None, :, b], [sums[:, b, h:h + 1] * mins[None, :, b, h] for h in range(mins.shape[2])]
        exact += dd * dw * i + sum(terms)
        if wtype in (11, 13):
            acc = r(dd * r(dw * i) + acc)
            if wtype == 13:
                acc = r(terms[0] + acc)
        else:
            v = r(terms[0])
            if wtype == 10:
                v = r(terms[1] + v)
            acc = r(r(dd * dw * i + v) + acc)
        if b % 8 == 7:
            s1 = r(total + acc)
            bb = r(s1 - total)
            low = r(low + r(r(total - r(s1 - bb)) + r(acc - bb)))
            total, acc = s1, torch.zeros_like(acc)
    return r(total + low).float(), exact


def _inputs32(kind, m, k, gen, dev):
    x = torch.randn(m, k, device=dev, generator=gen)
    if kind != "normal":
        x = x.abs()
    if kind == "one sign, a few large":
        x.view(m, -1, 32)[:, torch.randperm(k // 32, device=dev, generator=gen)[:k // 1024]] *= 50
    return x


# tiles on both sides of the border of the two sizes of the epilogue (32 | 48), ragged ones, a tile and a part of one, several per CTA; rows of outputs a multiple of
# 16 bytes apart (19000), of 8 (14340) and of 2 (19001)
@pytest.mark.parametrize("tokens,n,tile", [(16, 14340, 16), (31, 19000, 32), (33, 19001, 48), (50, 19000, 64), (61, 19001, 64), (100, 14340, 64), (130, 19001, 48)])
@pytest.mark.parametrize("wtype", sorted(NAMES))
def test_prompt32_tile_sizes_give_the_same_bits(lib, cuda_dev, tokens, n, tile, wtype):
    """A token's result does not depend on the size of the tile it is in: against few weight rows, for which tiles of 16 tokens are planned."""
    k = 512
    assert lib.cq_prompt32_tile_tokens(tokens, n) == tile and lib.cq_prompt32_tile_tokens(tokens, 200) == 16
    gen = torch.Generator(device=cuda_dev).manual_seed(n)
    wq, x = _weights32(wtype, n, k, 1.0, gen, cuda_dev)[0], torch.randn(tokens, k, device=cuda_dev, generator=gen)
    for dtype in (torch.float32, torch.float16, torch.bfloat16):
        out = _prompt32(lib, wtype, wq, x.to(dtype), k, n)
        for rows in (slice(0, 200), slice(n - 200, n)):
            assert torch.equal(out[:, rows], _prompt32(lib, wtype, wq[rows].contiguous(), x.to(dtype), k, 200))


@pytest.mark.parametrize("kind", ["normal", "one sign", "one sign, a few large"])
@pytest.mark.parametrize("tokens,k,n", [(9, 1024, 65), (33, 1280, 14336)])
@pytest.mark.parametrize("wtype", [3, 7])
def test_prompt32_sums_of_the_formats_with_a_minimum_per_block(lib, cuda_dev, wtype, tokens, k, n, kind):
    """Q4_1 and Q5_1, bit for bit: the chunks meet in an exact two-sum, whichever is the larger."""
    gen = torch.Generator(device=cuda_dev).manual_seed(k)
    wq, *parts = _weights32(wtype, n, k, 1.0, gen, cuda_dev)
    x = _inputs32(kind, tokens, k, gen, cuda_dev)
    assert torch.equal(_prompt32(lib, wtype, wq, x, k, n), _plain_sums(wtype, *parts, *_activations32(lib, wtype, x))[0])


@pytest.mark.parametrize("k", [1024, 4096])
@pytest.mark.parametrize("wtype", [6, 11])
def test_prompt32_is_no_further_from_64_bits_than_sums_per_block_where_chunks_differ(lib, cuda_dev, wtype, k):
    """The other formats with an exact two-sum.  3 % for the noise of 16384 values' errors."""
    gen = torch.Generator(device=cuda_dev).manual_seed(k)
    wq, *parts = _weights32(wtype, 256, k, 1.0, gen, cuda_dev)
    x = _inputs32("one sign, a few large", 64, k, gen, cuda_dev)
    plain, exact = _plain_sums(wtype, *parts, *_activations32(lib, wtype, x))
    err = lambda o: float((o.double() - exact).norm() / exact.norm())
    assert err(_prompt32(lib, wtype, wq, x, k, 256)) <= 1.03 * err(plain) <= 1e-6


@pytest.mark.parametrize("kind", ["normal", "one sign", "one sign, a few large"])
@pytest.mark.parametrize("minimum", [1.0, 0.0, -1.0, 8.0])
@pytest.mark.parametrize("k", [1024, 4096, 14336])
@pytest.mark.parametrize("wtype", [6, 10, 13])
def test_prompt32_minimum_sums_are_no_further_from_64_bits_than_sums_per_block(lib, cuda_dev, wtype, k, minimum, kind):
    """Minimum sums on the tensor core, also where they are most of the result and of one sign.  3 % for the noise of 16384 values' errors."""
    gen = torch.Generator(device=cuda_dev).manual_seed(k)
    wq, *parts = _weights32(wtype, 256, k, minimum, gen, cuda_dev)
    x = _inputs32(kind, 64, k, gen, cuda_dev)
    plain, exact = _plain_sums(wtype, *parts, *_activations32(lib, wtype, x))
    err = lambda o: float((o.double() - exact).norm() / exact.norm())
    assert err(_prompt32(lib, wtype, wq, x, k, 256)) <= 1.03 * err(plain) <= 1e-6


@pytest.mark.parametrize("wtype", [3, 6, 7, 10, 11, 13])
def test_prompt32_of_infinite_scales_and_inputs(lib, cuda_dev, wtype):
    """Results are not finite where the decode kernel's are not, and only there."""
    k, n, m, gen = 512, 96, 16, torch.Generator(device=cuda_dev).manual_seed(wtype)
    wq, x, st = _weights32(wtype, n, k, 1.0, gen, cuda_dev)[0].clone(), torch.randn(m, k, device=cuda_dev, generator=gen), torch.cuda.current_stream().cuda_stream
    x[2, 40], x[4, 300], x[6, 7], x[8, 100:140] = float("inf"), float("nan"), 1e9, -65000.0
    for row, at in ((5, MINIMUM[wtype][0]), (9, MINIMUM[wtype][1])):
        if at is not None:
            wq[row, at:at + 2] = torch.tensor([0, 0x7C], dtype=torch.uint8, device=cuda_dev)
    y8, decode = torch.zeros((m, k // 32, 36), dtype=torch.uint8, device=cuda_dev), torch.empty((m, n), device=cuda_dev)
    lib.cq_quantize_act(x.data_ptr(), capi.F32, y8.data_ptr(), k, k, m, 0, st)
    for r in range(0, m, 8):
        lib.cq_mmvq(wtype, 0, capi.F32, wq.data_ptr(), y8[r:].data_ptr(), decode[r:].data_ptr(), k, n, k // 32, n, 8, st)
    scratch, out = torch.zeros(lib.cq_prompt32_scratch_bytes(wtype, m, k), dtype=torch.uint8, device=cuda_dev), torch.empty((m, n), device=cuda_dev)
    lib.cq_prompt32_matmul(wtype, wq.data_ptr(), x.data_ptr(), capi.F32, out.data_ptr(), scratch.data_ptr(), k, n, m, n, st)
    capi.check("prompt32")
    ok = torch.isfinite(decode)
    assert torch.equal(torch.isfinite(out), ok) and not bool(ok[:, 5].any()) and bool(ok[0, 10:].all())
    assert float((out - decode)[ok].norm() / decode[ok].norm()) <= 2e-6


@pytest.mark.parametrize("wtype,rows,k,n", [(3, 200, 768, 700), (6, 200, 768, 700), (7, 200, 768, 700), (10, 200, 768, 700), (11, 200, 768, 700), (13, 200, 768, 700),
                                            (3, 40, 5120, 64), (13, 36, 5120, 64)])
def test_qmatmul_runs_the_kernel_the_rule_names(lib, oracle, cuda_dev, wtype, rows, k, n):
    """QMatMul.forward against both kernels called directly: the bits of the one the rule names, which differ from the other's."""
    _, x, wq = make_case(oracle, wtype, k, n, rows, seed=4)
    x_dev, w_dev, st = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev), torch.cuda.current_stream().cuda_stream
    prompt, kp = _prompt32(lib, wtype, w_dev, x_dev, k, n), capi.pad(k, 512)
    y8 = torch.zeros((rows, kp // 32, 36), dtype=torch.uint8, device=cuda_dev)
    lib.cq_quantize_act(x_dev.data_ptr(), capi.F32, y8.data_ptr(), k, kp, rows, 0, st)
    slices = torch.empty_like(prompt)
    for r in range(0, rows, 8):
        lib.cq_mmvq(wtype, 0, capi.F32, w_dev.data_ptr(), y8[r:].data_ptr(), slices[r:].data_ptr(), k, n, kp // 32, n, min(8, rows - r), st)
    capi.check("direct")
    y = QMatMul.from_qtensor(QTensor.from_data(wq, GgmlDType(wtype), (n, k), cuda_dev)).forward(x_dev)
    assert not torch.equal(prompt, slices)
    assert lib.cq_prompt32_pays(wtype, rows, k, n) == (1 if rows == 200 else 0)
    assert torch.equal(y, prompt if rows == 200 else slices)


def _at_offset(w_dev, offset):
    """The same bytes `offset` bytes into a larger buffer (whose base is 256-byte aligned)."""
    buf = torch.full((w_dev.numel() + 256,), 0xFF, dtype=torch.uint8, device=w_dev.device)
    buf[offset:offset + w_dev.numel()] = w_dev.reshape(-1)
    assert buf.data_ptr() % 256 == 0
    return buf[offset:offset + w_dev.numel()]


@pytest.mark.parametrize("wtype,offset", [(10, 2), (10, 4), (10, 6), (10, 14), (11, 2), (11, 4), (11, 6), (11, 14), (14, 4), (14, 8), (14, 12)])
@pytest.mark.parametrize("k,n,tokens", [(2048, 200, 40), (768, 129, 20)])
def test_weights_at_any_address_give_the_bits_of_an_aligned_copy(lib, oracle, cuda_dev, wtype, offset, k, n, tokens):
    """Bases off the 16-byte grid have no tensor map, and every row its own distance to the boundary below it."""
    _, x, wq = make_case(oracle, wtype, k, n, tokens, seed=offset)
    x_dev, w_dev = torch.from_numpy(x).to(cuda_dev), torch.from_numpy(wq).to(cuda_dev)
    run = _prompt if wtype == 14 else _prompt32
    assert torch.equal(run(lib, wtype, _at_offset(w_dev, offset), x_dev, k, n), run(lib, wtype, w_dev, x_dev, k, n))


def test_addresses_the_prompt_kernels_do_not_take_are_refused(lib, oracle, cuda_dev):
    """Q6_K off a 4-byte boundary, Q4_K and Q8_0 off a 16-byte one: an error before any launch, as before these kernels."""
    for wtype, offset in ((14, 2), (12, 8), (8, 8)):
        _, x, wq = make_case(oracle, wtype, 512, 64, 20, seed=1)
        w = _at_offset(torch.from_numpy(wq).to(cuda_dev), offset)
        mm = QMatMul.from_qtensor(QTensor.from_device_blocks(w, GgmlDType(wtype), (64, 512)))
        with pytest.raises(capi.CandleQError, match="aligned"):
            mm.forward(torch.from_numpy(x).to(cuda_dev))
        lib.cq_clear_status()


@pytest.mark.parametrize("wtype", [GgmlDType.Q4K, GgmlDType.Q6K, GgmlDType.Q8_0])
@pytest.mark.parametrize("n,pad,offset,tokens", [(136, 0, 0, 75), (136, 8, 0, 130), (136, 4, 0, 33), (136, 0, 1, 20), (129, 0, 0, 70), (135, 1, 0, 17), (8, 0, 0, 9), (260, 0, 0, 131)])
def test_16_bit_rows_at_any_distance(cuda_dev, wtype, n, pad, offset, tokens):
    """Rows of 16-bit outputs a multiple of 16 bytes apart (stored by eight) or not (a lane per row), ragged in rows and tokens: the f32 outputs
    rounded, and nothing between the rows."""
    _check_16_bit_rows(cuda_dev, wtype, n, pad, offset, tokens)


# tiles of several sizes (Q4_K and Q6_K | Q8_0), past the tile's first 64 (32) tokens and with an epilogue of either size
@pytest.mark.parametrize("wtype", [GgmlDType.Q4K, GgmlDType.Q6K, GgmlDType.Q8_0])
@pytest.mark.parametrize("n,pad,offset,tokens,tile,tile32", [(19000, 0, 0, 75, 80, 48), (19001, 0, 0, 75, 80, 48), (14340, 4, 0, 130, 80, 48), (19001, 2, 0, 61, 64, 64), (14340, 0, 0, 100, 112, 64),
                                                             (19000, 8, 0, 50, 64, 64), (14336, 0, 1, 100, 112, 64)])
def test_16_bit_rows_of_large_tiles(cuda_dev, wtype, n, pad, offset, tokens, tile, tile32):
    assert (capi.lib().cq_prompt32_tile_tokens(tokens, n) if wtype == GgmlDType.Q8_0 else capi.lib().cq_prompt_tile_tokens(int(wtype), tokens, n)) == \
        (tile32 if wtype == GgmlDType.Q8_0 else tile)
    _check_16_bit_rows(cuda_dev, wtype, n, pad, offset, tokens)


def _check_16_bit_rows(cuda_dev, wtype, n, pad, offset, tokens):
    from candle_b200.synth import random_blocks
    L, st, k, big = capi.lib(), torch.cuda.current_stream().cuda_stream, 512, wtype in (GgmlDType.Q4K, GgmlDType.Q6K)
    w = random_blocks(wtype, n, k, seed=n, device=cuda_dev)
    need = L.cq_prompt_scratch_bytes(tokens, k) if big else L.cq_prompt32_scratch_bytes(int(wtype), tokens, k)
    scratch = torch.empty(need, dtype=torch.uint8, device=cuda_dev)
    matmul = L.cq_prompt_matmul if big else L.cq_prompt32_matmul
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.randn(tokens, k, device=cuda_dev, generator=torch.Generator(device=cuda_dev).manual_seed(1)).to(dtype)
        out = []
        for xs in (x.float(), x):
            buf = torch.full((tokens * (n + pad) + 16,), -7.0, dtype=xs.dtype, device=cuda_dev)
            matmul(int(wtype), w.data_ptr(), xs.data_ptr(), ELEM[xs.dtype], buf[offset:].data_ptr(), scratch.data_ptr(), k, n, tokens, n + pad, st)
            capi.check("prompt")
            rows = buf[offset:offset + tokens * (n + pad)].view(tokens, n + pad)
            assert bool((rows[:, n:] == -7.0).all()) and bool((buf[:offset] == -7.0).all()) and bool((buf[offset + tokens * (n + pad):] == -7.0).all())
            out.append(rows[:, :n])
        assert torch.equal(out[0].to(dtype), out[1])


@pytest.mark.parametrize("wtype", [3, 6, 7, 10, 11, 13])
@pytest.mark.parametrize("tokens,k,n", [(16, 256, 128), (17, 768, 129), (75, 1280, 200), (130, 512, 300)])
def test_prompt32_bf16_results_are_neighbours(lib, oracle, cuda_dev, wtype, tokens, k, n):
    """The bf16 summation against the f32 sums of cq_prompt32_matmul, both within 1e-6 of the sums' 2-norm: a bf16 result is the rounded f32 one or its
    neighbour (2^-7 of the value at most), and hardly ever the latter (an interval of 4e-6 around boundaries 2^-8 apart, for small sums more)."""
    _, x, wq = make_case(oracle, wtype, k, n, tokens, seed=wtype)
    w_dev, xb = torch.from_numpy(wq).to(cuda_dev), torch.from_numpy(x).to(cuda_dev).to(torch.bfloat16)
    matmul = lambda t, wp, xp, _elem, out, scratch, kk, nn, m, stride, st: lib.cq_prompt32_bf16_matmul(t, wp, xp, out, scratch, kk, nn, m, stride, st)
    out = _run(lib.cq_prompt32_bf16_scratch_bytes(wtype, tokens, k), matmul, lib.cq_prompt32_timeout_flag, wtype, w_dev, xb, k, n).float()
    ref = _prompt32(lib, wtype, w_dev, xb.float(), k, n)
    slack = 4e-6 * float(ref.norm() / ref.numel() ** 0.5)
    assert bool(((out - ref.to(torch.bfloat16).float()).abs() <= 2.0 ** -7 * ref.abs() + slack).all())
    assert float((out != ref.to(torch.bfloat16).float()).float().mean()) <= 0.01


@pytest.mark.parametrize("tokens,k,n,offset", [(200, 768, 700, 0), (70, 1280, 129, 0), (40, 512, 14341, 0), (2000, 512, 2050, 0), (300, 8192, 1500, 0), (100, 1024, 999, 2)])
@pytest.mark.parametrize("wtype", [3, 6, 7, 10, 11, 13])
def test_qmatmul_bf16_prompts_are_the_sums_per_block(lib, cuda_dev, wtype, tokens, k, n, offset):
    """bf16 calls of the Q8_1 formats: the sums with a minimum added per block, rounded once, bit for bit; ragged rows and tokens, both tile sizes, weights
    at any even address for Q2_K and Q3_K."""
    gen = torch.Generator(device=cuda_dev).manual_seed(k + n)
    wq, *parts = _weights32(wtype, n, k, 1.0, gen, cuda_dev)
    x = torch.randn(tokens, k, device=cuda_dev, generator=gen).to(torch.bfloat16)
    w = wq.reshape(-1)
    if offset:
        w = _at_offset(w, offset if wtype in (10, 11) else 16)
    assert lib.cq_prompt32_bf16_pays(wtype, tokens, k, n) == 1
    y = QMatMul.from_qtensor(QTensor.from_device_blocks(w, GgmlDType(wtype), (n, k))).forward(x)
    assert torch.equal(y, _plain_sums(wtype, *parts, *_activations32(lib, wtype, x.float()))[0].to(torch.bfloat16))
    assert lib.cq_prompt32_timeout_flag() == 0 and lib.cq_prompt32_bf16_timeout_flag() == 0


@pytest.mark.parametrize("wtype,rows,k,n", [(3, 40, 5120, 64), (13, 36, 5120, 64), (10, 12, 14336, 3248), (6, 11, 8192, 1000)])
def test_qmatmul_bf16_rows_the_rule_leaves_to_the_decode_kernel(lib, cuda_dev, wtype, rows, k, n):
    gen = torch.Generator(device=cuda_dev).manual_seed(k)
    mm = QMatMul.from_qtensor(QTensor.from_device_blocks(_weights32(wtype, n, k, 1.0, gen, cuda_dev)[0].reshape(-1), GgmlDType(wtype), (n, k)))
    x = torch.randn(rows, k, device=cuda_dev, generator=gen).to(torch.bfloat16)
    assert lib.cq_prompt32_bf16_pays(wtype, rows, k, n) == 0
    assert torch.equal(mm.forward(x), torch.cat([mm.forward(x[r:r + 8]) for r in range(0, rows, 8)]))
