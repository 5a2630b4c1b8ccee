"""Host-side logic that needs no GPU: type registry, shape checks, error behaviour."""
import numpy as np
import pytest
import torch

from candle_b200 import capi
from candle_b200.quantized import GgmlDType, QMatMul, QTensor


def test_type_registry_matches_reference():
    """candle-core/src/quantized/mod.rs:300-342 (ids), :387-421 (sizes)."""
    ids = {"F32": 0, "F16": 1, "Q4_0": 2, "Q4_1": 3, "Q5_0": 6, "Q5_1": 7, "Q8_0": 8, "Q8_1": 9, "Q2K": 10,
           "Q3K": 11, "Q4K": 12, "Q5K": 13, "Q6K": 14, "Q8K": 15, "BF16": 30}
    for name, u in ids.items():
        assert GgmlDType.from_u32(u) is GgmlDType[name]
    with pytest.raises(capi.CandleQError, match="unknown dtype for tensor 4"):
        GgmlDType.from_u32(4)
    sizes = {"Q4_0": (18, 32), "Q8_0": (34, 32), "Q8_1": (36, 32), "Q4K": (144, 256), "Q6K": (210, 256),
             "Q8K": (292, 256), "Q2K": (84, 256), "Q3K": (110, 256), "Q5K": (176, 256), "Q4_1": (20, 32),
             "Q5_0": (22, 32), "Q5_1": (24, 32), "F32": (4, 1), "F16": (2, 1), "BF16": (2, 1)}
    for name, (ts, bs) in sizes.items():
        assert GgmlDType[name].type_size() == ts and GgmlDType[name].block_size() == bs


def test_oracle_and_library_agree_on_sizes(oracle):
    for name, code in (("Q4_0", capi.Q4_0), ("Q8_0", capi.Q8_0), ("Q4K", capi.Q4_K), ("Q6K", capi.Q6_K)):
        dt = getattr(oracle, name)
        assert oracle.TYPE_SIZE[dt] == capi.TYPE_SIZE[code] == GgmlDType(code).type_size()
        assert oracle.BLOCK_SIZE[dt] == capi.BLOCK_ELEMS[code] == GgmlDType(code).block_size()


@pytest.mark.skipif(torch.cuda.is_available(), reason="checks the no-GPU failure mode")
def test_fails_loudly_without_a_gpu(lib):
    """No CPU fallback: uploading weights or running a matmul without a CUDA device is an error."""
    blocks = np.zeros(4 * 144, dtype=np.uint8)
    with pytest.raises(capi.CandleQError):
        QTensor.from_data(blocks, GgmlDType.Q4K, (4, 256))
    with pytest.raises(capi.CandleQError, match="no CPU path"):
        QMatMul.__new__(QMatMul).forward(torch.zeros(1, 256))


def test_missing_library_is_an_error(monkeypatch, tmp_path):
    monkeypatch.setattr(capi, "_lib", None)
    monkeypatch.setattr(capi, "LIB_PATH", str(tmp_path / "nope.so"))
    with pytest.raises(capi.CandleQError, match="no CPU or PyTorch fallback"):
        capi.lib()


def test_moe_routing_matches_numpy_restatement():
    """fused_moe.rs:233-260: softmax, top-k (descending), renormalisation, pairs sorted by expert."""
    import numpy as np
    import torch
    from candle_b200.fused_moe import route, sort_pairs
    rng = np.random.default_rng(0)
    logits = rng.standard_normal((7, 16)).astype(np.float32)
    w, ids = route(torch.from_numpy(logits), 4, True)
    e = np.exp(logits - logits.max(-1, keepdims=True))
    p = e / e.sum(-1, keepdims=True)
    ref_ids = np.argsort(-p, axis=-1, kind="stable")[:, :4]
    ref_w = np.take_along_axis(p, ref_ids, -1)
    ref_w = ref_w / ref_w.sum(-1, keepdims=True)
    assert np.array_equal(ids.numpy(), ref_ids)
    assert np.allclose(w.numpy(), ref_w, rtol=1e-6, atol=1e-7)
    w2, _ = route(torch.from_numpy(logits), 4, False)
    assert np.allclose(w2.numpy(), np.take_along_axis(p, ref_ids, -1), rtol=1e-6, atol=1e-7)
    experts, pairs = sort_pairs(ids)
    flat = ref_ids.reshape(-1)
    assert np.array_equal(experts.numpy(), np.sort(flat, kind="stable"))
    assert np.array_equal(flat[pairs.numpy()], experts.numpy())          # pair indices in expert order
    assert sorted(pairs.tolist()) == list(range(flat.size))


def test_decoder_refuses_positions_beyond_max_pos():
    """The host-side bound of the decoder harness: claiming positions past max_pos raises before anything is launched
    (the KV cache and the rotary tables hold max_pos positions)."""
    import types

    import pytest

    from candle_b200.decoder import DecoderConfig, LlamaShapedDecoder
    stub = types.SimpleNamespace(cfg=DecoderConfig.tiny(), _pos_host=0)
    LlamaShapedDecoder._claim_positions(stub, 100)
    LlamaShapedDecoder._claim_positions(stub, 28)
    assert stub._pos_host == 128 == stub.cfg.max_pos
    with pytest.raises(ValueError, match="max_pos"):
        LlamaShapedDecoder._claim_positions(stub, 1)
    assert stub._pos_host == 128
    stub2 = types.SimpleNamespace(cfg=DecoderConfig.tiny(), _pos_host=0)
    with pytest.raises(ValueError, match="max_pos"):
        LlamaShapedDecoder.generate(stub2, __import__("torch").zeros((1, 120), dtype=__import__("torch").int64), 10)


def test_prompt_attention_is_taken_where_it_is_the_faster(lib):
    """(batch, queries, heads, cache) with the measured times of a CTA per query and of 32 queries per CTA (us, position 0 or the end
    of the cache): the slower kernel must not be taken.  Without a device the rule counts 148 SMs."""
    by_query = [((1, 17, 8, 1152), 21.4, 138.6), ((1, 17, 32, 1152), 54.7, 138.9), ((1, 21, 4, 1152), 13.4, 128.9), ((1, 26, 1, 1024), 13.4, 130.5),
                ((1, 25, 2, 640), 10.5, 85.4), ((2, 44, 8, 640), 40.0, 80.4), ((1, 32, 4, 64), 11.4, 25.1), ((1, 17, 16, 128), 9.3, 17.9),
                ((1, 95, 8, 896), 60.5, 116.3), ((1, 839, 2, 896), 81.6, 115.8), ((1, 912, 2, 1152), 112.8, 150.7), ((1, 64, 4, 1152), 26.9, 151.2)]
    by_32 = [((2, 512, 32, 640), 1181.1, 342.8), ((1, 1024, 32, 1152), 1609.2, 591.8), ((1, 256, 32, 256), 248.9, 78.2), ((1, 64, 32, 128), 60.4, 28.5),
             ((1, 128, 32, 1152), 309.1, 151.8), ((1, 512, 8, 512), 158.6, 76.3), ((4, 40, 16, 128), 71.3, 26.9)]
    for shape, slow, fast in by_query:
        assert slow < fast and lib.cq_attention_reads_by_32(*shape) == 0, shape
    for shape, slow, fast in by_32:
        assert fast < slow and lib.cq_attention_reads_by_32(*shape) == 1, shape
    assert lib.cq_attention_reads_by_32(2, 512, 32, 1161) == 0          # its scores do not fit shared memory
    assert lib.cq_attention_reads_by_32(64, 16, 64, 128) == 0


def test_operands_of_the_super_block_prompt_kernel_are_exact():
    """csrc/prompt_kq.cu: the f16 operands and the largest partial sum of every accumulator, for all scales and codes."""
    q, sc = np.meshgrid(np.arange(64), np.arange(-128, 128))
    y, prod = q - 32, (q - 32) * sc
    a = (prod + 12288).astype(np.float16).astype(np.int64) - 12288       # f32 -> f16 rounds as the fma does: the product is exact before it
    assert np.array_equal((1024 + q).astype(np.float16).astype(np.int64) - 1056, y)
    for part in (a, prod - a):
        assert np.array_equal(part.astype(np.float16).astype(np.int64), part)
    assert np.all(a % 8 == 0) and 256 * 128 * np.abs(a).max() <= 8 * 2 ** 24 and 256 * 128 * np.abs(prod - a).max() <= 2 ** 24
    # Q4_K: one accumulator per 128 elements, or per super-block up to the stored limit of sum |q8|
    assert 128 * 128 * 63 * 15 <= 2 ** 24 < 256 * 127 * 63 * 15 and (2 ** 24 // 945) * 945 <= 2 ** 24 and 16 * 63 * 2048 <= 2 ** 24


@pytest.mark.parametrize("rule,slices,prompt", [
    ("cq_prompt32_pays",
     [((7, 71, 10240, 53), 57.1, 83.9), ((3, 15, 8192, 7620), 41.8, 66.9), ((7, 34, 5120, 100), 25.9, 44.2), ((7, 11, 10240, 5467), 53.2, 86.1),
      ((7, 12, 14336, 6442), 77.0, 119.1), ((3, 10, 5120, 7202), 27.8, 44.0), ((10, 41, 5120, 34), 33.2, 43.6), ((6, 9, 768, 360), 7.6, 11.5),
      ((13, 18, 14336, 3248), 80.1, 101.7), ((13, 11, 8192, 7677), 55.9, 61.4), ((6, 11, 8192, 10496), 48.9, 71.8), ((11, 36, 5120, 128), 34.9, 48.2)],
     [((13, 512, 4096, 14336), 2235.0, 261.8), ((6, 91, 10240, 1629), 162.0, 87.3), ((3, 16, 768, 8303), 18.5, 11.8),
      ((10, 154, 10240, 171), 193.9, 83.4), ((3, 183, 14336, 496), 217.9, 114.2), ((6, 9, 512, 5178), 14.7, 9.8)]),
    ("cq_prompt32_bf16_pays",
     [((7, 71, 10240, 53), 56.9, 83.1), ((3, 15, 8192, 7620), 42.5, 67.3), ((7, 34, 5120, 100), 26.9, 44.1), ((7, 11, 10240, 5467), 54.2, 85.5),
      ((7, 12, 14336, 6442), 78.2, 118.0), ((3, 10, 5120, 7202), 28.6, 44.4), ((10, 41, 5120, 34), 34.6, 47.6), ((6, 9, 768, 360), 8.2, 11.3),
      ((13, 18, 14336, 3248), 80.9, 110.7), ((13, 11, 8192, 7677), 56.3, 66.6), ((6, 11, 8192, 10496), 49.5, 70.8), ((11, 36, 5120, 128), 37.4, 50.1)],
     [((13, 512, 4096, 14336), 2255.2, 330.1), ((6, 91, 10240, 1629), 169.7, 86.1), ((3, 16, 768, 8303), 19.2, 12.2),
      ((10, 154, 10240, 171), 198.2, 92.0), ((3, 183, 14336, 496), 226.9, 114.7), ((6, 9, 512, 5178), 15.0, 9.9)])])
def test_prompt_route_of_the_q8_1_formats_takes_the_faster_side(lib, rule, slices, prompt):
    """(type, tokens, K, rows) with the measured times of slices on the decode kernel and of the prompt kernel (us), f32 and bf16.  Without a device the
    rule counts 148 SMs."""
    for shape, fast, slow in slices:
        assert fast < slow and getattr(lib, rule)(*shape) == 0, shape
    for shape, slow, fast in prompt:
        assert fast < slow and getattr(lib, rule)(*shape) == 1, shape


def test_prompt_route_of_q6_k_takes_the_faster_kernel(lib):
    """(tokens, K, rows) with the measured times of the prompt kernel and of the int8 kernel (us)."""
    f16 = [((1154, 4096, 3648), 90.9, 110.2), ((24, 4096, 14208), 41.5, 58.0), ((393, 10240, 3587), 98.5, 133.9), ((512, 14336, 4096), 148.0, 170.0),
           ((707, 8192, 4800), 158.4, 229.5), ((65, 2048, 12091), 24.3, 37.7), ((25, 8704, 13177), 85.5, 108.5), ((51, 9728, 9856), 97.4, 117.5),
           ((1487, 4608, 9037), 293.0, 354.5)]
    int8 = [((18, 14336, 4096), 124.3, 90.8), ((61, 8192, 3210), 72.9, 62.3), ((899, 6144, 832), 64.1, 52.5), ((19, 14336, 1216), 120.3, 88.6),
            ((54, 11008, 5278), 106.6, 73.7), ((156, 2816, 512), 31.3, 25.5), ((196, 11776, 704), 113.1, 78.3), ((653, 12800, 4653), 267.9, 239.6)]
    for (tokens, k, n), fast, slow in f16:
        assert fast < slow and lib.cq_prompt_pays(14, tokens, k, n) == 1, (tokens, k, n)
    for (tokens, k, n), slow, fast in int8:
        assert fast < slow and lib.cq_prompt_pays(14, tokens, k, n) == 0, (tokens, k, n)
    assert lib.cq_prompt_pays(12, 18, 14336, 4096) == 1


def test_grouped_route_of_q6_k_takes_the_faster_kernel(lib):
    """(pairs, experts, rows) with the measured times of the int8 kernel and of the prompt kernel (us)."""
    int8 = [((320, 8, 768), 33.7, 45.7), ((396, 2, 1536), 33.6, 45.7), ((150, 2, 256), 25.6, 34.6), ((77 * 2, 8, 512), 33.3, 39.5)]
    f16 = [((432, 16, 512), 72.6, 52.0), ((832, 32, 256), 84.5, 58.0), ((8192, 128, 768), 220.2, 167.0), ((1024, 64, 1536), 195.6, 142.4),
           ((180, 16, 768), 42.1, 31.5)]
    for shape, fast, slow in int8:
        assert fast < slow and lib.cq_moe_prompt_pays(14, *shape) == 0, shape
    for shape, slow, fast in f16:
        assert fast < slow and lib.cq_moe_prompt_pays(14, *shape) == 1, shape
    assert lib.cq_moe_prompt_pays(12, 64, 2, 256) == 1


def test_shared_memory_of_another_cta_is_written_after_a_cluster_barrier():
    """Distributed shared memory may be written only once the CTA it belongs to runs: in every kernel the first remote address is made after a wait at
    the cluster's barrier (spelled out, or cluster_sync_all)."""
    import glob
    import os
    import re
    found = 0
    for path in glob.glob(os.path.join(os.path.dirname(capi.__file__), "csrc", "*.cu*")):
        for body in re.sub(r"//[^\n]*", "", open(path).read()).split("\n}\n"):      # one function each
            remote = re.search(r"cluster_map\(|mapa\.shared::cluster", body)
            if remote and "cluster_map(uint32_t" not in body:
                found += 1
                assert re.search(r"barrier\.cluster\.wait|cluster_sync_all\(\)", body[:remote.start()]), (path, body[:80])
    assert found >= 2
