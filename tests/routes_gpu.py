"""Which kernels a call runs: a rule that stopped taking the fast kernel, or took it where it must not, would pass every comparison of numbers.

Run by test_gpu_routes.py in a process of its own: in one that has launched thousands of kernels between two profiles, the profiler loses records."""
import json

import pytest
import torch

from oxibonsai_b200.runtime.observability import kernel_histogram

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def kernels(run) -> dict[str, int]:
    """Names of the kernels of one call of ``run`` and how often each was launched."""
    table = kernel_histogram(run, iterations=1)
    if not table:
        pytest.skip("the profiler recorded no device activity")
    return {name: row["count"] for name, row in table.items()}


def grids(run, part: str, tmp_path) -> list[list[int]]:
    """Grids of the launches of one call of ``run`` whose kernel's name holds ``part``."""
    from torch.profiler import ProfilerActivity, profile
    run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    out = [e["args"]["grid"] for e in events if part in e.get("name", "") and "grid" in e.get("args", {})]
    if not out and not any("grid" in e.get("args", {}) for e in events):
        pytest.skip("the profiler recorded no launches")
    return out


def launches(table: dict[str, int], part: str) -> int:
    return sum(n for name, n in table.items() if part in name)


@pytest.fixture(scope="module")
def wide_head_gguf(tmp_path_factory):
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    p = tmp_path_factory.mktemp("gguf") / "wide_head.gguf"
    write_synthetic_gguf(str(p), Qwen3Config(hidden=512, inter=1024, layers=2, heads=4, kv_heads=2, head_dim=128, vocab=1000, context=1024, name="wide"), seed=3)
    return str(p)


def engine(path, kv, max_batch=1, **kw):
    from oxibonsai_b200.runtime.engine import InferenceEngine
    return InferenceEngine(path, max_seq_len=1024, kv_dtype=kv, max_batch=max_batch, **kw)


@pytest.mark.parametrize("kv", ["q8", "q4"])
def test_exact_mode_multiplies_quantised_rows_in_f32(kv, wide_head_gguf):
    ran = {}
    for exact in (True, False):
        eng = engine(wide_head_gguf, kv, exact=exact)
        eng.open_sequence(list(range(1, 20)), 32, 0)
        ran[exact] = kernels(lambda: eng.runner.step_eager(1))
    assert launches(ran[True], "attn_decode") == 2 and not launches(ran[True], "attn_decode_quant")
    assert launches(ran[False], "attn_decode") == 2 == launches(ran[False], "attn_decode_quant")


@pytest.mark.parametrize("kv", ["q8", "q4"])
def test_exact_mode_verifies_quantised_rows_in_f32(kv, wide_head_gguf):
    """Drafted tokens go through a small chunk, whose attention is the decode kernel's (behind 300 tokens: no short INT4 prompt)."""
    ran = {}
    for exact in (True, False):
        eng = engine(wide_head_gguf, kv, exact=exact)
        eng._bind_slot(0, 400)
        drafted = torch.arange(1, 6, dtype=torch.int32, device=DEV)
        ran[exact] = kernels(lambda: eng.runner.verify_logits(drafted, 0, 300))
    assert launches(ran[True], "attn_decode") == 2 and not launches(ran[True], "attn_decode_quant")
    assert launches(ran[False], "attn_decode") == 2 == launches(ran[False], "attn_decode_quant")


@pytest.mark.parametrize("page,splits", [(8, 9), (64, 4)])
def test_splits_of_quantised_attention_follow_the_kernel(page, splits, tmp_path):
    """Pages of eight tokens stay on the CUDA cores, four CTAs an SM; the tensor-core kernel has two."""
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    path = str(tmp_path / "groups.gguf")
    write_synthetic_gguf(path, Qwen3Config(hidden=512, inter=1024, layers=1, heads=16, kv_heads=8, head_dim=128, vocab=1000, context=1024, name="groups"), seed=3)
    eng = engine(path, "q8", max_batch=8, page_size=page)
    for slot in range(8):
        eng.open_sequence(list(range(1, 20)), 32, slot)
    assert grids(lambda: eng.runner.step_eager(8), "attn_decode", tmp_path) == [[8, splits, 8]]


def test_threads_that_make_the_first_batch_product_together_get_the_same_rows():
    """The table of what the device holds is filled by the first call: in a process of its own, eight threads start with it at once."""
    import subprocess
    import sys
    code = """
import threading, torch
from oxibonsai_b200.ops import cuda_ops as K
dev = torch.device("cuda:0")
w = K.PlanarWeight(512, 1024, dev)
w.codes.random_(-2**31, 2**31 - 1)
w.scales.fill_(0.01)
x = torch.randn((5, 1024), device=dev).half()
K._gp()
torch.cuda.synchronize()
out, go = [None] * 8, threading.Barrier(8)
def run(i):
    torch.cuda.set_device(0)
    with torch.cuda.stream(torch.cuda.Stream()):
        y, st = torch.empty((5, 512), device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
        torch.cuda.current_stream().synchronize()
        go.wait()
        K.bitgemm_batch(w, x, out=y, status=st)
        torch.cuda.current_stream().synchronize()
        out[i] = y
threads = [threading.Thread(target=run, args=(i,)) for i in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
assert all(torch.equal(out[0], y) for y in out)
print("alike")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "alike" in r.stdout, r.stderr[-2000:]


def test_prompt_scratch_is_allocated_by_the_first_long_prompt(wide_head_gguf):
    """Decode steps, verification and short prompts run without it; where it does not fit, long prompts run without it too."""
    prompt = [int(t) for t in torch.randint(0, 1000, (200,), generator=torch.Generator().manual_seed(1))]
    tokens = []
    for room in (True, False):
        eng = engine(wide_head_gguf, "f16", max_batch=2)
        eng.open_sequence(prompt[:40], 64, 0)
        eng.open_sequence(prompt[:64], 80, 1)
        eng.step_batch([40, 64])
        eng.verify_greedy([1, 2, 3], 41)
        assert eng.runner._pf["wexp"] is None
        if not room:
            eng.runner._wexp_elems = lambda: 1 << 45
        tokens.append(eng.open_sequence(prompt, 300, 0))
        assert eng.runner._pf["wexp"].numel() == (eng.runner._wexp_elems() if room else 0)
        ran = kernels(lambda: eng.runner.prefill(torch.tensor(prompt, dtype=torch.int32, device=DEV), 0, 0))
        assert launches(ran, "expand_rows") == launches(ran, "gemm_pair") == (8 if room else 0) and launches(ran, "bitgemm_prefill") == (0 if room else 8)
        tokens.append(eng.runner.logits[0].clone())
    assert tokens[0] == tokens[2] and torch.equal(tokens[1], tokens[3])


@pytest.mark.parametrize("n", [20, 40, 65, 300, 1024, 1100])
def test_prefill_launches_counts_what_a_prompt_launches(n, wide_head_gguf):
    eng = engine(wide_head_gguf, "f16", max_batch=2)
    eng._bind_slot(0, 1024)
    tokens = torch.randint(0, 1000, (min(n, 1024),), dtype=torch.int32, device=DEV)
    pieces = [tokens] if n <= 1024 else [tokens, tokens[:n - 1024]]
    ran = sum(launches(kernels(lambda p=p: eng.runner.prefill(p, 0, 0)), "bonsai") for p in pieces)
    assert eng.runner.prefill_launches(n) == ran - (len(pieces) - 1) + 1


@pytest.mark.parametrize("batch", [1, 2, 3, 6])
def test_launches_of_a_block_format_step(batch, wide_head_gguf, tmp_path):
    """Products per pair of rows where the matrix is streamed."""
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    path = str(tmp_path / "wide_q8_0.gguf")
    cli.requantize_gguf(wide_head_gguf, path, "q8_0")
    eng = GenericQwen3Engine(path, max_seq_len=128, max_batch=6)
    for slot in range(batch):
        eng._bind(slot)
    ran = kernels(lambda: eng._forward(0, batch, True))
    products = launches(ran, "quant_stream") + launches(ran, "quant_gemv")
    assert products == 4 * eng.config.layers * -(-batch // 2)
    assert eng.kernel_launches_per_step(batch) == products + 5 * eng.config.layers + 4 + batch


@pytest.mark.parametrize("n", [65, 255, 256, 300])
def test_weights_expanded_slab_by_slab_give_the_same_prompt(n, tmp_path):
    """A scratch of 256 rows of the widest matrix: gate / up passes in slabs (the last one smaller) that overwrite one another, below 256 tokens
    the larger matrices stay packed.  Every sum runs in the same order, so logits and cache are those of one slab, bit for bit."""
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    path = str(tmp_path / "slabs.gguf")
    cfg = Qwen3Config(hidden=512, inter=1152, layers=2, heads=4, kv_heads=2, head_dim=128, vocab=1000, context=1024, name="slabs")
    write_synthetic_gguf(path, cfg, seed=5)
    prompt = [int(t) for t in torch.randint(0, 1000, (n,), generator=torch.Generator().manual_seed(n))]
    seen = []
    for small in (True, False):
        eng = engine(path, "f16")
        if small:
            eng.runner._wexp_elems = lambda: 256 * 1152
        eng.open_sequence(prompt, n + 8, 0)
        seen.append((eng.runner.logits[0].clone(), eng.kv.k.clone(), eng.kv.v.clone()))
        tokens = torch.tensor(prompt, dtype=torch.int32, device=DEV)
        ran = kernels(lambda: eng.runner.prefill(tokens, 0, 0))
        # rows of 512, 512, 512 and 1152 inputs: qkv 1024, o 512, gate / up 2304, down 512 of them
        slabs = (0 if n < 256 else 2) + 1 + (0 if n < 256 else 5) + (0 if n < 256 else 2) if small else 4
        packed = 3 if small and n < 256 else 0
        assert launches(ran, "expand_rows") == launches(ran, "gemm_pair") == 2 * slabs and launches(ran, "bitgemm_prefill") == 2 * packed
    for a, b in zip(*seen):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kvt,page,hd,scratch,order,tensor_memory", [(1, 64, 128, 0, 0, True), (1, 16, 128, 0, 0, False), (1, 128, 128, 0, 0, True), (1, 64, 64, 0, 0, False), (1, 64, 128, 0, 1, False),
                                                                    (0, 64, 128, 0, 0, False), (2, 16, 128, 2 * 2 * 128 * 256, 0, True), (3, 64, 128, 2 * 2 * 128 * 256, 0, True),
                                                                    (2, 64, 128, 2 * 2 * 128 * 256 - 1, 0, False), (3, 64, 128, 0, 0, False)])
def test_prompt_attention_takes_the_kernel_of_its_form(kvt, page, hd, scratch, order, tensor_memory):
    from oxibonsai_b200.ops import cuda_ops as K
    T, nkv = 200, 2
    q, pages = torch.randn((T, 4, hd), device=DEV), -(-T // page)
    row = hd // 2 if kvt == 3 else hd
    pools = [torch.zeros((pages, nkv, page, row), dtype=K.KV_DTYPES[kvt], device=DEV) for _ in range(2)]
    scales = [torch.ones((pages, nkv, page), device=DEV) if kvt >= 2 else None for _ in range(2)]
    table = torch.arange(pages, dtype=torch.int32, device=DEV)
    room = torch.empty(scratch, dtype=torch.float16, device=DEV) if scratch else None
    ran = kernels(lambda: K.attn_prefill(q, 0, table, 4, nkv, hd, kvt, page, *pools, *scales, k_order=order, scratch=room))
    assert launches(ran, "attn_prefill_tc") == int(tensor_memory) and launches(ran, "attn_prefill") == 1
    assert launches(ran, "kv_to_f16") == int(tensor_memory and kvt >= 2)


@pytest.mark.parametrize("kvt,page,nq,part", [(1, 64, 4, "attn_decode_mma"), (2, 64, 4, "attn_decode_quant"), (3, 16, 16, "attn_decode_quant"), (2, 8, 4, "attn_decode_h128"), (3, 24, 4, "attn_decode_kernel"),
                                              (2, 8, 16, "attn_decode_kernel"), (0, 64, 4, "attn_decode_kernel")])
def test_decode_attention_takes_the_kernel_of_its_form(kvt, page, nq, part):
    from oxibonsai_b200.ops import cuda_ops as K
    nkv, pages = 2, 4
    pools = [torch.zeros((pages, nkv, page, 64 if kvt == 3 else 128), dtype=K.KV_DTYPES[kvt], device=DEV) for _ in range(2)]
    scales = [torch.ones((pages, nkv, page), device=DEV) if kvt >= 2 else None for _ in range(2)]
    table, pos = torch.arange(pages, dtype=torch.int32, device=DEV)[None], torch.tensor([20], dtype=torch.int32, device=DEV)
    q = torch.randn((1, nq, 128), device=DEV)
    ran = kernels(lambda: K.attn_decode(q, pos, table, nq, nkv, 128, kvt, page, *pools, *scales, nsplit=4))
    assert launches(ran, "attn_decode") == 1 == launches(ran, part)
