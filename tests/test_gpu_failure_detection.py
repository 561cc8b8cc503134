"""Failure detection of the tensor-parallel kernels on one GPU, without any fault: a communicator whose peer never
writes makes every bounded wait run out; the kernel must return, record its status code and leave the context usable."""
import numpy as np
import pytest
import torch

from oxibonsai_b200.core import TQ2_0_G128, quantize

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda:0")


def test_barrier_wait_expires_with_status_3():
    from oxibonsai_b200.ops import cuda_ops as K
    from oxibonsai_b200.parallel.tp import TpGroup
    tp = TpGroup.loopback(_dev(), size=2)
    tp.set_spin_limit(2000)
    tp.barrier()
    torch.cuda.synchronize()
    assert tp.status() == 3
    with pytest.raises(K.CudaKernelError):
        tp.check()
    # the context is alive and other kernels still run
    assert float(torch.ones(8, device=_dev()).sum()) == 8.0
    tp.close()


@pytest.mark.parametrize("fast", [True, False])
def test_fused_gemv_allreduce_reports_a_silent_peer(fast):
    from oxibonsai_b200.ops import cuda_ops as K
    from oxibonsai_b200.parallel.tp import TpGroup, _lib
    rows, cols = 256, 512
    rng = np.random.default_rng(0)
    raw = quantize(TQ2_0_G128, (rng.standard_normal((rows, cols)) * 0.05).astype(np.float32))
    pw = K.PlanarWeight(rows, cols, _dev()).fill_from_gguf(torch.from_numpy(raw).to(_dev()), TQ2_0_G128, cols, 0, rows)
    tp = TpGroup.loopback(_dev(), size=2, hidden=rows)
    tp.set_spin_limit(2000)
    word = torch.zeros(1, dtype=torch.int32, device=_dev())
    tp.use_status_word(word)
    x = torch.randn(cols, device=_dev())
    res = torch.randn(rows, device=_dev())
    out = torch.empty(rows, device=_dev())
    if fast:
        K.bitgemv_s16(K.S16Weight(pw), x, epi=K.EPI_TP, residual=res, out=out, comm=tp.handle, status=word)
    else:
        K.check(_lib().bonsai_bitgemv_tp(tp.handle, pw.codes.data_ptr(), pw.scales.data_ptr(), x.data_ptr(), 1e-6, out.data_ptr(),
                                         res.data_ptr(), rows, cols, 0, K.stream()), "bitgemv_tp")
    torch.cuda.synchronize()
    assert int(word.item()) == 2
    # the kernel returned: the exchange counter moved on, so a later healthy exchange would not be confused with this one
    assert int(tp.state[0].item()) == 1
    tp.close()


def test_engine_raises_when_the_status_word_is_set(tiny_gguf):
    """A non-zero status word read with the sampled token turns into CudaKernelError instead of a token."""
    from oxibonsai_b200.ops import cuda_ops as K
    from oxibonsai_b200.runtime import EngineBuilder
    eng = EngineBuilder().model_path(tiny_gguf).preset("greedy").max_seq_len(64).build()
    assert eng.generate([1, 2, 3], 2)            # healthy
    it = eng.generate_stream([1, 2, 3], 4)
    next(it)
    eng.runner.status.fill_(2)                   # what a kernel does when a peer stays silent
    with pytest.raises(K.CudaKernelError):
        for _ in it:
            pass
    assert int(eng.runner.status.item()) == 0    # cleared once reported
    assert eng.generate([1, 2, 3], 2)            # and the engine is usable again


@pytest.mark.parametrize("call", ["prompt", "batch", "verification"])
def test_expired_waits_of_prompts_batches_and_verification_are_reported(call, tiny_gguf):
    """The word that the tensor-core GEMMs of these passes record an expired wait in is the one that is read with the tokens."""
    from oxibonsai_b200.ops import cuda_ops as K
    from oxibonsai_b200.runtime import EngineBuilder
    eng = EngineBuilder().model_path(tiny_gguf).preset("greedy").max_seq_len(128).max_batch(2).build()
    prompt = list(range(1, 41))
    eng.open_sequence(prompt, 64, 0)
    eng.open_sequence(prompt, 64, 1)
    pass_of = {"prompt": lambda: eng.open_sequence(prompt, 64, 0), "batch": lambda: eng.step_batch([40, 40]), "verification": lambda: eng.verify_greedy([3, 4, 5], 40)}[call]
    assert pass_of()
    eng.runner._pf["status"].fill_(1)            # what a GEMM does whose pipeline stalls
    with pytest.raises(K.CudaKernelError, match="stalled"):
        pass_of()
    assert int(eng.runner.status.item()) == 0 and pass_of()


def test_expired_waits_of_block_format_prompts_are_reported(tiny_gguf, tmp_path, monkeypatch):
    import torch
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    from oxibonsai_b200.ops import cuda_ops as K
    path = str(tmp_path / "tiny_q8_0.gguf")
    cli.requantize_gguf(tiny_gguf, path, "q8_0")
    eng = GenericQwen3Engine(path, max_seq_len=128, max_batch=2)
    prompt = list(range(1, 41))

    def first_token(slot):
        eng.begin_sequence(prompt, 64, slot)
        eng.prefill_slot(prompt, slot)
        return eng.finish_sequence(prompt, slot)

    good = [first_token(0), first_token(1)]
    product = K.dense_gemm_f16

    def stalled(*args, status=None, **kw):
        out = product(*args, status=status, **kw)
        status.fill_(1)
        return out

    monkeypatch.setattr(K, "dense_gemm_f16", stalled)
    with pytest.raises(K.CudaKernelError, match="stalled"):
        first_token(1)
    monkeypatch.setattr(K, "dense_gemm_f16", product)
    assert [first_token(0), first_token(1)] == good and len(eng.step_batch([40, 40])) == 2
    torch.cuda.synchronize()


def test_prompt_attention_takes_a_status_word(tiny_gguf):
    """The tensor-memory kernel has waits that can expire: it is given the word in which the products of the same prompt record theirs, and
    leaves it alone when all is well.  Its code has a text of its own."""
    from oxibonsai_b200.models.slot_state import SlotState
    from oxibonsai_b200.ops import cuda_ops as K
    dev, T, nkv = _dev(), 200, 2
    q = torch.randn((T, 4, 128), device=dev)
    pools = [torch.randn((4, nkv, 64, 128), device=dev).half() for _ in range(2)]
    table, status = torch.arange(4, dtype=torch.int32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    a = K.attn_prefill(q, 0, table, 4, nkv, 128, K.KV_F16, 64, *pools, status=status)
    assert int(status.item()) == 0 and torch.equal(a, K.attn_prefill(q, 0, table, 4, nkv, 128, K.KV_F16, 64, *pools))
    assert "attention" in SlotState.STATUS_TEXT[6]


def test_streamed_rows_take_the_status_word_of_the_engine(tiny_gguf, tmp_path, monkeypatch):
    """Every product of a block-format decode step records an expired wait where the engine reads it with the tokens."""
    from oxibonsai_b200 import cli
    from oxibonsai_b200.models.qwen3_generic import GenericQwen3Engine
    from oxibonsai_b200.ops import cuda_ops as K
    path = str(tmp_path / "tiny_q8_0.gguf")
    cli.requantize_gguf(tiny_gguf, path, "q8_0")
    eng = GenericQwen3Engine(path, max_seq_len=64, max_batch=2)
    words, product = [], K.quant_gemv_batched
    monkeypatch.setattr(K, "quant_gemv_batched", lambda *a: (words.append(a[-1]), product(*a))[1])
    eng._bind(0)
    eng._forward(0, 1, True)
    assert len(words) == 4 * eng.config.layers and all(w is eng.status for w in words) and eng._read_tokens(1)
    eng.status.fill_(5)
    with pytest.raises(K.CudaKernelError, match="copy pipeline"):
        eng.step_batch([1])
    assert eng.step_batch([1])
