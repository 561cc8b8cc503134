"""Generic-format GPU path: the block-decoding GEMV for every GGUF type and a whole model served from Q8_0 / Q4_K / FP8."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oxibonsai_b200.core import gguf as G

TYPES = [("F32", G.F32, 1e-5), ("F16", G.F16, 1e-5), ("BF16", G.BF16, 1e-5), ("Q4_0", G.Q4_0, 1e-5), ("Q8_0", G.Q8_0, 1e-5), ("TQ2_0", G.TQ2_0, 1e-5),
         ("F8_E4M3", G.F8_E4M3, 1e-5), ("F8_E5M2", G.F8_E5M2, 1e-5), ("Q2_K", G.Q2_K, 1e-5), ("Q3_K", G.Q3_K, 1e-5), ("Q4_K", G.Q4_K, 1e-5),
         ("Q5_K", G.Q5_K, 1e-5), ("Q6_K", G.Q6_K, 1e-5), ("Q8_K", G.Q8_K, 1e-5)]


@pytest.mark.parametrize("name,tid,tol", TYPES)
def test_quant_gemv_matches_fp32_reference_of_the_decoded_matrix(name, tid, tol):
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(3)
    n, k = 77, 1024
    w = rng.normal(size=(n, k)).astype(np.float32) * 0.05
    q = quantize(tid, w)
    wd = torch.from_numpy(dequantize(tid, q).reshape(n, k)).double()
    x = torch.from_numpy(rng.normal(size=k).astype(np.float32))
    nw = torch.from_numpy(rng.uniform(0.5, 1.5, k).astype(np.float32))
    res = torch.from_numpy(rng.normal(size=n).astype(np.float32))
    qd = torch.from_numpy(q).to(dev)
    y = K.quant_gemv(tid, qd, n, k, x.to(dev)).cpu().double()
    ref = wd @ x.double()
    assert (y - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item()) * 10, name
    xn = nw * x * torch.rsqrt((x * x).mean() + 1e-6)
    y2 = K.quant_gemv(tid, qd, n, k, x.to(dev), norm_w=nw.to(dev), eps=1e-6, residual=res.to(dev)).cpu().double()
    ref2 = wd @ xn.double() + res.double()
    assert torch.allclose(y2, ref2, rtol=1e-4, atol=1e-4), name


def test_swiglu_kernel():
    from oxibonsai_b200.ops import cuda_ops as K
    g, u = torch.randn(5000, device="cuda:0"), torch.randn(5000, device="cuda:0")
    assert torch.allclose(K.swiglu(g, u), torch.nn.functional.silu(g) * u, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("fmt", ["q8_0", "q4_k", "f8_e4m3"])
def test_generic_engine_follows_the_cpu_oracle(fmt, tiny_gguf, tmp_path):
    from oxibonsai_b200 import cli
    from oxibonsai_b200.core import GgufFile, Oracle
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    path = str(tmp_path / f"tiny_{fmt}.gguf")
    cli.requantize_gguf(tiny_gguf, path, fmt)
    prompt = [11, 257, 3, 999, 42, 7, 100, 5]
    want, _ = Oracle(GgufFile.open(path), 128).generate_greedy(prompt, 12)
    eng = GenericQwen3Engine(path, max_seq_len=128, kv_dtype="f32")
    got = eng.generate(prompt, 12, stop_at_eos=False)
    agree = sum(a == b for a, b in zip(got, want))
    assert len(got) == 12 and agree >= 10, (fmt, got, want)      # f32 everywhere; only the summation order differs from the CPU
    assert eng.generate(prompt, 12, stop_at_eos=False) == got     # graph replay is deterministic
    assert eng.kernel_launches_per_step() == 9 * 2 + 5       # fused Q/K/V and gate/up: 9 launches per layer


@pytest.mark.parametrize("name,tid,tol", TYPES)
def test_quant_to_f16_decodes_every_block_format(name, tid, tol):
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(5)
    n, k = 37, 512
    q = quantize(tid, rng.normal(size=(n, k)).astype(np.float32) * 0.05)
    want = torch.from_numpy(dequantize(tid, q).reshape(n, k)).to(dev).half()      # the kernel rounds the same f32 value once
    qd = torch.from_numpy(q).to(dev)
    nat = K.quant_to_f16(tid, qd, n, k, paired=False)
    assert torch.allclose(nat.float(), want.float(), rtol=2e-3, atol=1e-6), name      # one f16 ulp: the device may fuse d * q - m
    paired = K.quant_to_f16(tid, qd, n, k, paired=True)
    perm = K.paired_k_index(k, dev)
    assert torch.equal(paired[:, perm], nat), name
    # dense GEMM over paired-K operands with the residual epilogue against fp32 PyTorch
    x = torch.randn(70, k, device=dev)
    res = torch.randn(70, n, device=dev)
    got = K.dense_gemm_f16(paired, K.norm_to_f16_paired(x, None), residual=res)
    ref = res + x.half().float() @ nat.float().T
    assert torch.allclose(got, ref, rtol=1e-3, atol=1e-3), name


@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
def test_generic_engine_tensor_core_prompt_path_matches_token_by_token(fmt, tiny_gguf, tmp_path):
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    path = str(tmp_path / f"tiny_{fmt}.gguf")
    cli.requantize_gguf(tiny_gguf, path, fmt)
    prompt = [int(t) for t in np.random.default_rng(9).integers(0, 1000, 90)]
    slow = GenericQwen3Engine(path, max_seq_len=256, kv_dtype="f32", prefill_min=10**9)
    fast = GenericQwen3Engine(path, max_seq_len=256, kv_dtype="f32", prefill_min=16, prefill_chunk=64)   # two chunks, the second ragged
    assert fast.prefill_supported()
    a = slow.generate(prompt, 1, stop_at_eos=False)
    b = fast.generate(prompt, 1, stop_at_eos=False)
    la, lb = slow.logits[0].float(), fast.logits[0].float()
    assert torch.nn.functional.cosine_similarity(la, lb, dim=0).item() > 0.999, fmt     # f16 operands in the prompt path only
    assert (la - lb).abs().max().item() <= 0.03 * la.abs().max().item(), fmt
    n = len(prompt) - 1
    ka = slow.kpool[:, : (n + 63) // 64].float()
    kb = fast.kpool[:, : (n + 63) // 64].float()
    assert torch.allclose(ka, kb, rtol=2e-2, atol=2e-2)
    assert len(a) == 1 and len(b) == 1


def test_engine_builder_routes_checkpoints_by_weight_format(tiny_gguf, tmp_path):
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    from oxibonsai_b200.runtime import EngineBuilder, SamplingPreset
    from oxibonsai_b200.runtime.engine import GenericFormatEngine, InferenceEngine
    path = str(tmp_path / "tiny_q8_0.gguf")
    cli.requantize_gguf(tiny_gguf, path, "q8_0")
    eng = EngineBuilder().model_path(path).preset("greedy").max_seq_len(128).kv_cache("f32").build()
    assert isinstance(eng, GenericFormatEngine)
    prompt = [11, 257, 3, 999, 42, 7, 100, 5]
    got = eng.generate(prompt, 6, stop_at_eos=False)
    want = GenericQwen3Engine(path, max_seq_len=128, kv_dtype="f32").generate(prompt, 6, SamplingPreset.GREEDY.params(), stop_at_eos=False)
    assert got == want and len(got) == 6
    assert eng.last_stats.prompt_tokens == 8 and eng.last_stats.generated_tokens == 6 and eng.last_stats.decode_tokens_per_second > 0
    info = eng.model_info()
    assert info["weight_format"].upper().startswith("Q8_0") and info["weight_bytes"] > 0 and info["layers"] == 2
    assert eng.generate_seeded(prompt, 4, seed=7) == eng.generate_seeded(prompt, 4, seed=7)
    assert isinstance(EngineBuilder().model_path(tiny_gguf).max_seq_len(64).build(), InferenceEngine)


@pytest.mark.parametrize("name,tid", [("Q4_0", G.Q4_0), ("Q8_0", G.Q8_0), ("Q4_K", G.Q4_K), ("Q6_K", G.Q6_K), ("F8_E4M3", G.F8_E4M3), ("F16", G.F16)])
@pytest.mark.parametrize("batch", [2, 3, 8, 11])
def test_batched_quant_gemv_matches_fp32_reference(name, tid, batch):
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(11)
    n, k = 70, 1024
    q = quantize(tid, rng.normal(size=(n, k)).astype(np.float32) * 0.05)
    wd = torch.from_numpy(dequantize(tid, q).reshape(n, k)).double()
    x = torch.from_numpy(rng.normal(size=(batch, k)).astype(np.float32))
    nw = torch.from_numpy(rng.uniform(0.5, 1.5, k).astype(np.float32))
    res = torch.from_numpy(rng.normal(size=(batch, n)).astype(np.float32))
    qd = torch.from_numpy(q).to(dev)
    y = K.quant_gemv_batched(tid, qd, n, k, x.to(dev)).cpu().double()
    assert torch.allclose(y, x.double() @ wd.T, rtol=1e-4, atol=1e-4), name
    xn = nw * x * torch.rsqrt((x * x).mean(dim=1, keepdim=True) + 1e-6)
    # output and residual as column ranges of a wider buffer, as the fused projections use them
    wide = torch.zeros((batch, n + 16), device=dev)
    wide[:, 8:8 + n] = res.to(dev)
    K.quant_gemv_batched(tid, qd, n, k, x.to(dev), norm_w=nw.to(dev), eps=1e-6, residual=wide[:, 8:8 + n], out=wide[:, 8:8 + n])
    assert torch.allclose(wide[:, 8:8 + n].cpu().double(), xn.double() @ wd.T + res.double(), rtol=1e-4, atol=1e-4), name
    assert wide[:, :8].abs().max().item() == 0.0 and wide[:, 8 + n:].abs().max().item() == 0.0


def test_swiglu_rows_kernel():
    from oxibonsai_b200.ops import cuda_ops as K
    gu = torch.randn(5, 2 * 300 + 4, device="cuda:0")[:, : 2 * 300]
    want = torch.nn.functional.silu(gu[:, :300]) * gu[:, 300:]
    assert torch.allclose(K.swiglu_rows(gu, 300), want, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
def test_generic_engine_batched_decode_through_the_scheduler(fmt, tiny_gguf, tmp_path):
    """Several sequences decoded together by the generic-format engine (batched GEMV, batch attention and sampler) give the
    streams of the same sequences decoded alone; slots are compacted when a sequence ends early."""
    from oxibonsai_b200 import cli
    from oxibonsai_b200.runtime import EngineBuilder, SamplingPreset
    from oxibonsai_b200.runtime.scheduler import BatchScheduler
    path = str(tmp_path / f"tiny_{fmt}.gguf")
    cli.requantize_gguf(tiny_gguf, path, fmt)
    eng = EngineBuilder().model_path(path).preset("greedy").max_seq_len(160).max_batch(4).kv_cache("f32").build()
    assert eng.max_batch == 4 and eng.model_info()["max_batch"] == 4
    rng = np.random.default_rng(4)
    prompts = [[int(t) for t in rng.integers(0, 1000, n)] for n in (9, 30, 5, 21, 12)]
    lens = [12, 6, 10, 8, 9]
    greedy = SamplingPreset.GREEDY.params()
    alone = [eng.generate(p, n, greedy, stop_at_eos=False) for p, n in zip(prompts, lens)]
    sched = BatchScheduler(eng, eos_token=-1).start()
    try:
        reqs = [sched.submit(p, greedy, n) for p, n in zip(prompts, lens)]
        got = [r.wait(timeout=120) for r in reqs]
    finally:
        sched.stop()
    assert [len(g) for g in got] == lens
    agree = sum(x == y for a, b in zip(alone, got) for x, y in zip(a, b))
    assert agree >= sum(lens) - 2, (alone, got)       # f32 everywhere; the batched GEMV only changes nothing but launch shapes
    assert eng.kv_utilization() == 0.0


def test_standalone_rmsnorm_and_residual_add():
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(5, 2560, generator=g).to(dev), (torch.rand(2560, generator=g) + 0.5).to(dev)
    ref = x * torch.rsqrt((x * x).mean(dim=1, keepdim=True) + 1e-6) * w
    assert torch.allclose(K.rmsnorm(x, w, 1e-6), ref, rtol=1e-5, atol=1e-6)
    assert torch.allclose(K.rmsnorm(x[0], None, 1e-6), x[0] * torch.rsqrt((x[0] * x[0]).mean() + 1e-6), rtol=1e-5, atol=1e-6)
    wide = torch.randn(3, 300, generator=g).to(dev)
    view = wide[:, :128]                                       # rows with a stride
    assert torch.allclose(K.rmsnorm(view, None), view * torch.rsqrt((view * view).mean(dim=1, keepdim=True) + 1e-6), rtol=1e-5, atol=1e-6)
    a, b = torch.randn(100003, generator=g).to(dev), torch.randn(100003, generator=g).to(dev)
    want = a + b
    assert torch.equal(K.residual_add(a, b), want)


@pytest.mark.parametrize("name,tid,tol", TYPES)
@pytest.mark.parametrize("n,k", [(8, 256), (44, 2560), (1201, 2560), (600, 4096), (24, 12288), (16, 16384), (16, 16640)])
def test_streamed_rows_of_every_format(name, tid, tol, n, k):
    """Few rows, odd row counts (whose bytes cannot be copied in 16-byte units for some formats), widths that leave lanes of the last warp
    idle, the widest matrix that is streamed and one beyond it; one to three tokens."""
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(n + k)
    q = quantize(tid, rng.normal(size=(n, k)).astype(np.float32) * 0.05)
    wd = torch.from_numpy(dequantize(tid, q).reshape(n, k)).double()
    qd = torch.from_numpy(q).to(dev)
    nw = torch.from_numpy(rng.uniform(0.5, 1.5, k).astype(np.float32))
    for batch in (1, 2, 3):
        x = torch.from_numpy(rng.normal(size=(batch, k)).astype(np.float32))
        res = torch.from_numpy(rng.normal(size=(batch, n)).astype(np.float32))
        y = K.quant_gemv_batched(tid, qd, n, k, x.to(dev), norm_w=nw.to(dev), eps=1e-6, residual=res.to(dev)).cpu().double()
        xn = nw.double() * x.double() * torch.rsqrt((x.double() ** 2).mean(dim=1, keepdim=True) + 1e-6)
        # every sum runs over at most K / 32 + 64 rounded steps of terms whose magnitudes add up to |x| |W|, with minima taken off separately
        terms = xn.abs() @ wd.abs().T * (3.0 if name in ("Q2_K", "Q4_K", "Q5_K") else 1.0) + res.abs()
        assert ((y - (xn @ wd.T + res.double())).abs() <= 2.0 ** -23 * (k / 32 + 64) * terms).all(), (name, batch)


@pytest.mark.parametrize("tid", [G.Q4_0, G.Q8_0, G.Q4_K])
@pytest.mark.parametrize("n,k,batch", [(16, 256, 1), (77, 512, 1), (2000, 2560, 1), (28700, 256, 1), (300, 9728, 1), (24, 12288, 1), (24, 12544, 1),
                                       (24000, 256, 2), (23437, 256, 2), (2347, 2560, 3), (490, 12288, 2)])
def test_rows_of_exact_block_products(tid, n, k, batch):
    """Tiles of sixteen rows that end inside the matrix, several tiles and segments per CTA, the widest rows and one beyond, matrices on both sides
    of the least for two tokens; block inputs of very different size, zero blocks, inputs that are not finite."""
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(n + k + batch)
    few = quantize(tid, rng.normal(size=(8, k)).astype(np.float32) * 0.05).reshape(8, -1)
    pick = rng.integers(0, 8, n)
    wd, qd = torch.from_numpy(dequantize(tid, few.reshape(-1)).reshape(8, k)[pick]).double(), torch.from_numpy(few[pick].copy()).to(dev)
    x = rng.normal(size=(batch, k)).astype(np.float32) * np.exp2(rng.integers(-60, 3, (batch, k // 32)).repeat(32, 1)).astype(np.float32)
    x[:, 32:64] = 0
    x[:, 64:256:37] = 3e4
    room = torch.zeros(batch, k + 8)
    room[:, :k] = torch.from_numpy(x)
    y = K.quant_gemv_batched(tid, qd, n, k, room.to(dev)[:, :k]).cpu().double()
    xd = torch.from_numpy(x).double()
    # inputs are held to 2^-28 of their block's largest, the sums run over at most 64 rounded steps
    # of terms whose magnitudes add up to |x| |W| (three times that where minima are taken off separately)
    held = xd.abs().view(batch, -1, 32).amax(2).repeat_interleave(32, 1) * 2.0 ** -28
    terms = (xd.abs() * (64 * 2.0 ** -24) + held) @ wd.abs().T * (3.0 if tid == G.Q4_K else 1.0)
    assert ((y - xd @ wd.T).abs() <= terms).all()
    for bad in (float("nan"), float("inf")):
        room[0, k - 1] = bad
        y = K.quant_gemv_batched(tid, qd, n, k, room.to(dev)[:, :k])
        assert not torch.isfinite(y[0]).any() and torch.isfinite(y[1:]).all()
        if bad == float("inf") and tid != G.Q4_K:          # (minima come off separately: infinity minus infinity)
            assert torch.equal(y[0].cpu().nan_to_num(7.0), (wd[:, k - 1].float() * bad).nan_to_num(7.0))


@pytest.mark.parametrize("tid", [G.Q4_0, G.Q8_0, G.Q4_K])
@pytest.mark.parametrize("n,k,batch", [(48, 512, 1), (2000, 4096, 2), (300, 9728, 1), (24576, 256, 2)])
@pytest.mark.parametrize("size", [2.0 ** 16, 2.0 ** 31, 2.0 ** 33, 1e20])
def test_block_rows_keep_inputs_beside_an_outlier(tid, n, k, batch, size):
    """An outlier whose codes are zero leaves its neighbours every bit they have: sizes that the inputs' terms span, the largest they do, and
    two beyond, whose blocks are multiplied in f32."""
    from oxibonsai_b200.core.blocks import dequantize, quantize
    from oxibonsai_b200.ops import cuda_ops as K
    rng = np.random.default_rng(n + k)
    src = rng.normal(size=(8, k)).astype(np.float32) * 0.05
    if tid == G.Q4_K:
        src = np.abs(src)                # no minima: code zero is weight zero
    src[:, 5::96] = 0
    few = quantize(tid, src).reshape(8, -1)
    pick = rng.integers(0, 8, n)
    wd, qd = torch.from_numpy(dequantize(tid, few.reshape(-1)).reshape(8, k)[pick]).double(), torch.from_numpy(few[pick].copy()).cuda()
    assert not wd[:, 5::96].any()
    x = rng.normal(size=(batch, k)).astype(np.float32)
    x[:, 5::96] = size
    y = K.quant_gemv_batched(tid, qd, n, k, torch.from_numpy(x).cuda()).cpu().double()
    xd = torch.from_numpy(x).double()
    # at most 64 rounded steps of terms whose magnitudes add up to |x| |W|
    assert ((y - xd @ wd.T).abs() <= 64 * 2.0 ** -24 * (xd.abs() @ wd.abs().T)).all()


@pytest.mark.parametrize("tid", [G.Q4_0, G.Q8_0, G.Q4_K])
@pytest.mark.parametrize("n,k", [(16, 256), (1000, 2560), (2048, 2048), (2343, 2560), (2344, 2560), (620, 9728), (490, 12288), (480, 12544)])
def test_a_row_of_a_batch_is_the_row_alone(tid, n, k):
    """Sequences come and go beside one another without moving results: the same bits alone, as one of a pair and as the last of an odd batch, on both
    sides of the sizes at which the streamed kernels change."""
    from oxibonsai_b200.core.blocks import quantize
    from oxibonsai_b200.ops import cuda_ops as K
    rng = np.random.default_rng(n)
    few = quantize(tid, rng.normal(size=(8, k)).astype(np.float32) * 0.05).reshape(8, -1)
    w = torch.from_numpy(few.view(np.uint8).reshape(8, -1)[rng.integers(0, 8, n)].copy()).cuda()
    x, norm = (torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda() for s in ((3, k), (k,)))
    x[1, ::64] *= 1e12
    both = K.quant_gemv_batched(tid, w, n, k, x, norm, 1e-6)
    for b in range(3):
        assert torch.equal(both[b], K.quant_gemv_batched(tid, w, n, k, x[b:b + 1], norm, 1e-6)[0]), b
        assert torch.equal(both[b], K.quant_gemv(tid, w, n, k, x[b], norm, 1e-6)), b


@pytest.mark.parametrize("name,tid,tol", TYPES)
@pytest.mark.parametrize("n,k", [(1, 256), (3, 512), (77, 1280)])
def test_rows_decoded_from_whole_words_are_those_of_single_values(name, tid, tol, n, k):
    """Warps of 32 blocks that cross rows and end early, the last block of a matrix; a matrix at an odd address keeps the kernel that reads bytes."""
    from oxibonsai_b200.core.blocks import quantize
    from oxibonsai_b200.ops import cuda_ops as K
    rng = np.random.default_rng(n)
    raw = torch.from_numpy(quantize(tid, rng.normal(size=(n, k)).astype(np.float32) * 0.05).reshape(-1).view(np.uint8).copy()).cuda()
    room = torch.empty(raw.numel() + 8, dtype=torch.uint8, device="cuda")
    room[4:4 + raw.numel()] = raw
    for paired in (True, False):
        assert torch.equal(K.quant_to_f16(tid, raw, n, k, paired=paired), K.quant_to_f16(tid, room[4:4 + raw.numel()], n, k, paired=paired)), name


@pytest.mark.parametrize("fmt", ["q8_0", "q4_k"])
@pytest.mark.parametrize("kv", ["f16", "q4"])
def test_native_prompt_chunk_leaves_the_bits_of_its_kernels_one_by_one(fmt, kv, tiny_gguf, tmp_path):
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    path = str(tmp_path / f"tiny_{fmt}.gguf")
    cli.requantize_gguf(tiny_gguf, path, fmt)
    tokens = torch.from_numpy(np.random.default_rng(9).integers(0, 1000, 150).astype(np.int32)).cuda()
    caches = []
    for slabs in (None, 1, 0):
        eng = GenericQwen3Engine(path, max_seq_len=256, kv_dtype=kv, prefill_chunk=100)
        eng._bind(0)
        buffers = eng._prompt_buffers(0)
        if slabs == 1:                       # half of the gate and up rows at a time
            c = eng.config
            buffers["scratch"] = buffers["scratch"][:max(c.hidden * c.inter, c.heads * c.head_dim * c.hidden, (c.heads + 2 * c.kv_heads) * c.head_dim * c.hidden)]
        if slabs is None:
            for at in (0, 100):
                eng._short_chunk(tokens[at:at + 100], at, 0, buffers["scratch"])
        else:
            eng.prefill(tokens, 0, 0)
        caches.append([t.clone() for t in (eng.kpool, eng.vpool, eng.kscale, eng.vscale) if t is not None])
    for other in caches[1:]:
        assert all(torch.equal(a, b) for a, b in zip(caches[0], other))


def _token_by_token(path, prompt, **kw):
    """Logits and cache of an engine that feeds the prompt through the decode step."""
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    eng = GenericQwen3Engine(path, prefill_min=10**9, **kw)
    eng.generate(prompt, 1, stop_at_eos=False)
    return eng


@pytest.mark.parametrize("hidden,inter,heads", [(128, 256, 4), (128, 128, 1), (256, 128, 8)])
def test_prompts_of_narrow_models(hidden, inter, heads, tmp_path):
    """Matrices of fewer rows than a slab of the scratch matrix, which they fit as a whole."""
    from oxibonsai_b200 import cli
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    cfg = Qwen3Config(hidden=hidden, inter=inter, layers=2, heads=heads, kv_heads=1, head_dim=128, vocab=512, context=256, name="narrow")
    write_synthetic_gguf(str(tmp_path / "a.gguf"), cfg, tied=False, seed=3)
    path = str(tmp_path / "b.gguf")
    cli.requantize_gguf(str(tmp_path / "a.gguf"), path, "q8_0")
    prompt = [int(t) for t in np.random.default_rng(1).integers(0, 500, 100)]
    slow = _token_by_token(path, prompt, max_seq_len=128, kv_dtype="f32")
    fast = GenericQwen3Engine(path, max_seq_len=128, kv_dtype="f32")
    assert fast.prefill_supported() and len(fast.generate(prompt, 1, stop_at_eos=False)) == 1
    la, lb = slow.logits[0], fast.logits[0]
    assert (la - lb).abs().max().item() <= 0.03 * la.abs().max().item()          # f16 operands in the prompt path only


def test_prompts_pay_for_the_chunks_that_run(tiny_gguf, tmp_path):
    """Short prompts allocate no more than one matrix and what they free again; longer ones activations of their length, also when the chunks are
    made longer behind the first."""
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    from oxibonsai_b200.ops import cuda_ops as K
    path = str(tmp_path / "tiny_q8_0.gguf")
    cli.requantize_gguf(tiny_gguf, path, "q8_0")
    prompt = [int(t) for t in np.random.default_rng(9).integers(0, 1000, 400)]
    eng = GenericQwen3Engine(path, max_seq_len=448)
    c = eng.config
    K.gemm_workspace(eng.device)

    def grown(n):
        before = torch.cuda.memory_allocated()
        eng.begin_sequence(prompt[:n], n + 1, 0)
        eng.prefill_slot(prompt[:n], 0)
        eng.finish_sequence(prompt[:n], 0)
        logits = eng.logits[0].clone()
        eng.close_sequence(0)
        return torch.cuda.memory_allocated() - before, logits

    grown(2)                                  # the last token's step has buffers of its own
    matrix = 2 * max(c.hidden * c.inter, c.heads * c.head_dim * c.hidden)
    token = 16 * c.hidden + 8 * (c.heads + c.kv_heads) * c.head_dim + 4 * c.heads * c.head_dim + 2 * c.inter + 1024
    first, short = grown(41)
    assert first <= matrix + (64 << 10)
    assert grown(101)[0] <= matrix + 100 * token + (64 << 10)
    eng.prefill_chunk = 100
    want = grown(400)[1]
    eng.prefill_chunk = 399
    _, got = grown(400)
    assert torch.nn.functional.cosine_similarity(want, got, dim=0).item() > 0.999 and torch.equal(grown(41)[1], short)


def _requantise_by_name(src, dst, choose):
    """``src`` with every matrix in the block type that ``choose`` gives its name."""
    from oxibonsai_b200.core import GgufFile, GgufWriter, dequantize, quantize
    f, w = GgufFile.open(src), GgufWriter()
    for k, v in f.metadata.items():
        w.add(k, v)
    for t in f.tensors:
        raw = f.tensor_bytes(t.name)
        if len(t.dims) == 2 and not t.name.endswith("norm.weight"):
            tid = choose(t.name)
            w.add_tensor(t.name, t.dims, tid, quantize(tid, dequantize(t.type, raw) if t.type != G.F32 else np.frombuffer(raw, dtype=np.float32)))
        else:
            w.add_tensor(t.name, t.dims, t.type, np.frombuffer(raw, dtype=np.uint8))
    w.write(dst)
    return dst


MIXED = {"blk.0.attn_v": G.Q6_K, "blk.0.ffn_up": G.Q4_K, "blk.1.attn_q": G.Q4_0, "blk.1.attn_k": G.Q5_K, "blk.1.ffn_gate": G.F8_E4M3, "blk.1.ffn_down": G.BF16}


@pytest.mark.parametrize("kv", ["f32", "f16", "q8"])
@pytest.mark.parametrize("mixed", [False, True])
def test_native_prompt_chunks_match_token_by_token(kv, mixed, tiny_gguf, tmp_path):
    """Two native chunks and the last token's native step, over every page format whose codes do not hang on the last digits; matrices of one type side by
    side, and layers in which Q / K / V or gate / up are of different types."""
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    path = _requantise_by_name(tiny_gguf, str(tmp_path / "a.gguf"), lambda name: MIXED.get(name.removesuffix(".weight"), G.Q8_0) if mixed else G.Q8_0)
    prompt = [int(t) for t in np.random.default_rng(9).integers(0, 1000, 190)]
    slow = _token_by_token(path, prompt, max_seq_len=256, kv_dtype=kv)
    fast = GenericQwen3Engine(path, max_seq_len=256, kv_dtype=kv, prefill_chunk=100)
    assert [len(w["qkv"]) for w in fast.layers] == ([2, 3] if mixed else [1, 1]) and [len(w["gate_up"]) for w in fast.layers] == ([2, 2] if mixed else [1, 1])
    fast.generate(prompt, 1, stop_at_eos=False)
    la, lb = slow.logits[0], fast.logits[0]
    assert torch.nn.functional.cosine_similarity(la, lb, dim=0).item() > 0.999          # f16 operands in the prompt path only
    assert (la - lb).abs().max().item() <= 0.03 * la.abs().max().item()


@pytest.mark.parametrize("kv", ["f16", "q8", "q4"])
def test_the_last_token_of_a_prompt_runs_the_matrices_of_a_decode_step(kv, tmp_path):
    """Query and key rows in one matrix beside values of another type (how K-quant checkpoints are made), of sizes at which the pair and the single
    matrices have different kernels: the same bits as the decode step, in logits and cache."""
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    cfg = Qwen3Config(hidden=2048, inter=256, layers=2, heads=16, kv_heads=8, head_dim=128, vocab=512, context=128, name="mixed")
    write_synthetic_gguf(str(tmp_path / "a.gguf"), cfg, tied=False, seed=3)
    path = _requantise_by_name(str(tmp_path / "a.gguf"), str(tmp_path / "b.gguf"), lambda name: G.Q8_0 if "attn_v" in name else G.Q4_0)
    caches = []
    for native in (True, False):
        eng = GenericQwen3Engine(path, max_seq_len=64, kv_dtype=kv)
        eng._bind(0)
        assert [m.n for m in eng.layers[0]["qkv"]] == [3072, 1024]
        for i, t in enumerate((5, 300, 17)):
            eng.token[0], eng.pos[0] = t, i
            eng._forward_row(0) if native else eng._forward(0, 1, False)
        caches.append([t.clone() for t in (eng.logits, eng.kpool, eng.vpool, eng.kscale, eng.vscale) if t is not None])
    assert all(torch.equal(a, b) for a, b in zip(*caches))


def test_expired_waits_of_native_prompt_chunks_are_reported(tiny_gguf, tmp_path, monkeypatch):
    """The status word that a native chunk is given is the one that the engine reads with the prompt's first token."""
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    from oxibonsai_b200.ops import cuda_ops as K
    eng = GenericQwen3Engine(_requantise_by_name(tiny_gguf, str(tmp_path / "a.gguf"), lambda name: G.Q8_0), max_seq_len=256, max_batch=2)
    prompt = [int(t) for t in np.random.default_rng(9).integers(0, 1000, 120)]

    def first_token(slot):
        eng.begin_sequence(prompt, 130, slot)
        eng.prefill_slot(prompt, slot)
        return eng.finish_sequence(prompt, slot)

    good = [first_token(0), first_token(1)]
    chunk = K.blocks_prompt_chunk

    def stalled(prompt, layers, *args):
        chunk(prompt, layers, *args)
        assert eng.status.data_ptr() in list(prompt)
        eng.status.fill_(1)              # what a product of the chunk does whose pipeline stalls

    monkeypatch.setattr(K, "blocks_prompt_chunk", stalled)
    with pytest.raises(K.CudaKernelError, match="stalled"):
        first_token(1)
    monkeypatch.setattr(K, "blocks_prompt_chunk", chunk)
    assert [first_token(0), first_token(1)] == good


@pytest.mark.parametrize("first", [40, 70])
def test_prompt_buffers_outlive_the_stream_that_uses_them(first, tiny_gguf, tmp_path):
    """Buffers that one stream allocated and another still uses when a longer prompt replaces them are not handed out meanwhile."""
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    eng = GenericQwen3Engine(_requantise_by_name(tiny_gguf, str(tmp_path / "a.gguf"), lambda name: G.Q8_0), max_seq_len=256)
    eng._bind(0)
    tokens = torch.arange(1, 201, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        eng.prefill(tokens[:first])
        torch.cuda.synchronize()
    old = [eng._wscratch] if first <= 64 else [eng._prompt[k] for k in ("tokens", "h", "q", "act")]
    used = [(t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in old]
    sizes = [t.numel() * t.element_size() for t in old]
    del old
    with torch.cuda.stream(b):
        torch.cuda._sleep(1 << 30)                 # half a second
        eng.prefill(tokens[:first])
        eng.prefill(tokens)
        waiting = torch.cuda.Event()
        waiting.record()
    with torch.cuda.stream(a):
        taken = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(16)]
    assert not waiting.query()
    assert not any(t.data_ptr() < hi and lo < t.data_ptr() + t.numel() for t in taken for lo, hi in used)
    torch.cuda.synchronize()
