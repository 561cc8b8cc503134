"""Prefill kernels (tcgen05 GEMM with in-smem weight expansion, causal paged attention) against fp32 references."""
import numpy as np
import pytest
import torch

from oxibonsai_b200.core import Q1_0_G128, TQ2_0_G128, dequantize, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _random_quant(ty, rows, cols, seed):
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((rows, cols)) * 0.05).astype(np.float32)
    raw = quantize(ty, w)
    return raw, torch.from_numpy(dequantize(ty, raw).reshape(rows, cols))


def test_paired_k_layout_round_trip():
    from oxibonsai_b200.ops import cuda_ops as K
    x = torch.randn(3, 256, device=DEV)
    y = K.norm_to_f16_paired(x)
    perm = K.paired_k_index(256, DEV)
    assert torch.equal(y[:, perm], x.half())
    w = torch.rand(256, device=DEV) + 0.5
    yn = K.norm_to_f16_paired(x, w, 1e-6)
    ref = w * x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    assert torch.allclose(yn[:, perm].float(), ref, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("ty", [TQ2_0_G128, Q1_0_G128])
@pytest.mark.parametrize("rows,cols,T", [(256, 256, 64), (6144, 4096, 300), (1000, 2560, 256), (512, 12288, 513), (4096, 1024, 1),
                                         (128, 12288, 7), (4096, 12288, 64), (24576, 4096, 33), (200, 128, 5), (640, 384, 65)])
def test_bitgemm_prefill_matches_fp32(ty, rows, cols, T):
    from oxibonsai_b200.ops import cuda_ops as K
    raw, wd = _random_quant(ty, rows, cols, 21)
    pw = K.PlanarWeight(rows, cols, DEV).fill_from_gguf(torch.from_numpy(raw).to(DEV), ty, cols, 0, rows)
    g = torch.Generator().manual_seed(22)
    x = torch.randn(T, cols, generator=g)
    xp = K.norm_to_f16_paired(x.to(DEV))
    ref = x.half().double() @ wd.double().T
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    y = K.bitgemm_prefill(pw, xp, status=st)
    assert st.item() == 0
    scale = ref.abs().max().item()
    assert (y.cpu().double() - ref).abs().max().item() <= 2e-4 * scale
    res = torch.randn(T, rows, generator=g)
    y = K.bitgemm_prefill(pw, xp, epi=1, residual=res.to(DEV), status=st)
    assert (y.cpu().double() - (ref + res.double())).abs().max().item() <= 2e-4 * scale + 1e-5
    y16 = K.bitgemm_prefill(pw, xp, epi=3, status=st)
    assert (y16.cpu().double() - ref).abs().max().item() <= 2e-3 * scale
    if rows % 32 == 0:
        ys = K.bitgemm_prefill(pw, xp, epi=2, status=st)
        want = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
        perm = K.paired_k_index(rows // 2)
        got = ys.cpu()[:, perm].double()
        assert (got - want).abs().max().item() <= 3e-3 * want.abs().max().item() + 1e-4
    assert st.item() == 0
    # the balanced distribution sums partial tiles in a fixed order: repeatable bit for bit, and close to whole tiles
    y1 = K.bitgemm_prefill(pw, xp, status=st, balanced=True)
    y2 = K.bitgemm_prefill(pw, xp, status=st, balanced=True)
    y0 = K.bitgemm_prefill(pw, xp, status=st, balanced=False)
    assert torch.equal(y1, y2) and st.item() == 0
    assert (y1 - y0).abs().max().item() <= 5e-5 * scale
    assert int(K.gemm_workspace(DEV)[:65536].view(torch.int32).abs().sum().item()) == 0   # counters back to zero


@pytest.mark.parametrize("kvt,tol", [(1, 4e-3), (0, 3e-3), (2, 3e-2)])
@pytest.mark.parametrize("nq,nkv,hd,T,pos0", [(8, 2, 128, 100, 0), (4, 4, 64, 64, 37), (4, 1, 128, 200, 130)])
def test_attn_prefill_matches_reference(kvt, tol, nq, nkv, hd, T, pos0):
    from oxibonsai_b200.core.oracle import rope_table
    from oxibonsai_b200.ops import cuda_ops as K
    page, eps = 16, 1e-6
    total = pos0 + T
    npages = (total + page - 1) // page
    g = torch.Generator().manual_seed(31)
    kfull, vfull = torch.randn(total, nkv, hd, generator=g), torch.randn(total, nkv, hd, generator=g)
    q = torch.randn(T, nq, hd, generator=g)
    row = {0: hd, 1: hd, 2: hd}[kvt]
    kpool = torch.zeros((npages, nkv, page, row), dtype=K.KV_DTYPES[kvt], device=DEV)
    vpool = torch.zeros_like(kpool)
    ksc = torch.zeros((npages, nkv, page), device=DEV) if kvt >= 2 else None
    vsc = torch.zeros((npages, nkv, page), device=DEV) if kvt >= 2 else None
    perm_pages = torch.randperm(npages, generator=g)
    bt = perm_pages.to(torch.int32).to(DEV)
    kd, vd = kfull.clone(), vfull.clone()
    for t in range(total):
        pg, sl = int(perm_pages[t // page]), t % page
        for pool, sc, src, dst in ((kpool, ksc, kfull, kd), (vpool, vsc, vfull, vd)):
            if kvt == 2:
                s = src[t].abs().amax(-1) / 127
                qv = torch.round(src[t] / s[:, None]).clamp(-127, 127)
                pool[pg, :, sl] = qv.to(torch.int8).to(DEV)
                sc[pg, :, sl] = s.to(DEV)
                dst[t] = qv * s[:, None]
            else:
                pool[pg, :, sl] = src[t].to(K.KV_DTYPES[kvt]).to(DEV)
                dst[t] = src[t].to(K.KV_DTYPES[kvt]).float()
    out = K.attn_prefill(q.to(DEV), pos0, bt, nq, nkv, hd, kvt, page, kpool, vpool, ksc, vsc)
    perm = K.paired_k_index(nq * hd)
    got = out.cpu()[:, perm].float().view(T, nq, hd)
    grp = nq // nkv
    kk, vv = kd.repeat_interleave(grp, 1), vd.repeat_interleave(grp, 1)     # [total, nq, hd]
    sc_ = torch.einsum("tnd,snd->nts", q, kk) / hd ** 0.5
    mask = torch.arange(total)[None, :] <= (pos0 + torch.arange(T))[:, None]
    sc_ = sc_.masked_fill(~mask[None], float("-inf"))
    ref = torch.einsum("nts,snd->tnd", torch.softmax(sc_, -1), vv)
    assert (got - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item())
    if (nq * hd) % 128 == 0:        # the same rows in the K order of the mma.sync GEMM
        out_h = K.attn_prefill(q.to(DEV), pos0, bt, nq, nkv, hd, kvt, page, kpool, vpool, ksc, vsc, k_order=1)
        assert torch.equal(out_h.cpu()[:, K.hmma_k_index(nq * hd)], out.cpu()[:, perm])


@pytest.mark.parametrize("rows,cols,T", [(151936, 2048, 3), (1000, 4096, 64), (300, 256, 200)])
def test_dense_f16_gemm_on_tcgen05(rows, cols, T):
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator().manual_seed(41)
    w = (torch.randn(rows, cols, generator=g) * 0.02).half().to(DEV)
    x = torch.randn(T, cols, generator=g).half().to(DEV)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    y = K.dense_gemm_f16(w, x, status=st)
    ref = x.float() @ w.float().T
    assert st.item() == 0
    assert (y - ref).abs().max().item() <= 2e-3 * ref.abs().max().item()


@pytest.mark.parametrize("ty", [TQ2_0_G128, Q1_0_G128])
@pytest.mark.parametrize("rows,cols,T", [(6144, 4096, 64), (4096, 4096, 33), (24576, 4096, 64), (4096, 12288, 64), (512, 2560, 5), (200, 128, 1),
                                         (1000, 384, 16), (256, 9728, 17)])
def test_bitgemm_hmma_matches_fp32(ty, rows, cols, T):
    """Decode-batch GEMM on mma.sync with register-expanded weights, against a plain fp32 matmul of the same operands."""
    from oxibonsai_b200.ops import cuda_ops as K
    raw, wd = _random_quant(ty, rows, cols, 41)
    pw = K.PlanarWeight(rows, cols, DEV).fill_from_gguf(torch.from_numpy(raw).to(DEV), ty, cols, 0, rows)
    g = torch.Generator().manual_seed(42)
    x = torch.randn(T, cols, generator=g)
    xh = K.norm_to_f16_hmma(x.to(DEV))
    perm = K.hmma_k_index(cols)
    assert torch.equal(xh.cpu()[:, perm], x.half())           # the layout is a pure permutation
    ref = x.half().double() @ wd.double().T
    scale = ref.abs().max().item()
    y = K.bitgemm_hmma(pw, xh)
    assert (y.cpu().double() - ref).abs().max().item() <= 2e-4 * scale
    res = torch.randn(T, rows, generator=g)
    y = K.bitgemm_hmma(pw, xh, epi=1, residual=res.to(DEV))
    assert (y.cpu().double() - (ref + res.double())).abs().max().item() <= 2e-4 * scale + 1e-5
    nw = torch.rand(cols, generator=g) + 0.5
    xn = nw * x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    xnh = K.norm_to_f16_hmma(x.to(DEV), nw.to(DEV), 1e-6)
    assert torch.allclose(xnh.cpu()[:, perm].float(), xn, rtol=2e-3, atol=2e-3)
    if rows % 256 == 0:
        ys = K.bitgemm_hmma(pw, xh, epi=2)
        want = torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]
        got = ys.cpu()[:, K.hmma_k_index(rows // 2)].double()
        assert (got - want).abs().max().item() <= 3e-3 * want.abs().max().item() + 1e-4


@pytest.mark.parametrize("ty", [TQ2_0_G128, Q1_0_G128])
def test_expanded_rows_are_the_decoded_weights(ty):
    from oxibonsai_b200.ops import cuda_ops as K
    n, k = 77, 384
    raw, want = _random_quant(ty, n, k, 5)
    w = K.PlanarWeight(n, k, torch.device(DEV))
    w.fill_from_gguf(torch.from_numpy(np.array(raw, copy=True)).to(DEV), ty, k, 0, n)
    want = want.half()
    perm = K.paired_k_index(k)
    for row0, rows in ((0, n), (5, 1), (40, 37)):
        assert torch.equal(K.expand_rows(w, row0, rows).cpu()[:, perm], want[row0:row0 + rows])


@pytest.mark.parametrize("rows,cols,T,tile", [(1, 64, 1, 0), (130, 64, 33, 32), (256, 192, 256, 256), (300, 320, 257, 0), (514, 4096, 77, 48), (1024, 448, 700, 240)])
@pytest.mark.parametrize("sms", [2, 6, 148])
def test_pair_gemm_matches_fp64(rows, cols, T, tile, sms):
    """Remainders of rows (256 per tile), tokens (any multiple of 16 per tile) and stages (six 64-input blocks), one cluster for all
    tiles and one for each."""
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator(device=DEV).manual_seed(rows + T)
    w = (torch.randn((rows, cols), device=DEV, generator=g) * cols ** -0.5).half()
    x = torch.randn((T, cols), device=DEV, generator=g).half()
    res = torch.randn((T, rows), device=DEV, generator=g)
    want, terms = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    # products are exact in f32; every addition of the accumulator may drop one unit in the last place
    bound = 2.0 ** -23 * (cols + 4) * (terms + res.abs().double())
    a, b = (K.gemm_pair(w, x, e, residual=r, status=status, sms=sms, tile_tokens=tile) for e, r in ((0, None), (1, res)))
    assert ((a.double() - want).abs() <= bound).all() and ((b.double() - want - res.double()).abs() <= bound).all()
    half = 2.0 ** -11
    assert ((K.gemm_pair(w, x, 3, status=status, sms=sms, tile_tokens=tile).double() - want).abs() <= bound + half * want.abs() + 2.0 ** -25).all()
    if rows % 2 == 0:
        gate, up = want[:, 0::2], want[:, 1::2]
        act = torch.nn.functional.silu(gate) * up
        n = rows // 2
        wide = torch.zeros((T, (n + 15) // 16 * 16), dtype=torch.float16, device=DEV)      # paired-K order moves inputs within eight
        K.gemm_pair(w, x, 2, out=wide, status=status, sms=sms, tile_tokens=tile)
        got = wide[:, K.paired_k_index(wide.shape[1], DEV)][:, :n].double()
        # |d silu| <= 1.1 |d gate|; the fast exponential and division add 2^-20
        slack = 1.1 * bound[:, 0::2] * up.abs() + gate.abs() * bound[:, 1::2] + (half + 2.0 ** -20) * act.abs() + 2.0 ** -24
        assert ((got - act).abs() <= slack).all()
    assert status.item() == 0


@pytest.mark.parametrize("rows", [300, 302, 306, 320])
def test_pair_gemm_gated_units_stay_inside_their_rows(rows):
    """SwiGLU rows in paired-K order take whole groups of eight: the output has room for them, and a row without it is refused."""
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator(device=DEV).manual_seed(rows)
    w, x = (torch.randn(s, device=DEV, generator=g).half() for s in ((rows, 256), (70, 256)))
    out = K.gemm_pair(w, x, epi=2)
    unit, width = rows // 2, (rows // 2 + 7) // 8 * 8
    assert out.shape == (70, width)
    gate, up = (x.double() @ w[i::2].double().T for i in range(2))
    want = torch.nn.functional.silu(gate) * up
    got = torch.zeros((70, (width + 15) // 16 * 16), dtype=torch.float16, device=DEV)
    got[:, :width] = out
    got = got[:, K.paired_k_index(got.shape[1], DEV)][:, :unit].double()
    assert ((got - want).abs() <= 2.0 ** -10 * want.abs() + 1e-3).all()
    if width != unit:
        with pytest.raises(K.CudaKernelError):
            K.gemm_pair(w, x, epi=2, out=torch.empty((70, unit), dtype=torch.float16, device=DEV))


@pytest.mark.parametrize("nq,nkv,T,pos0,kvt,page", [(3, 3, 1, 0, 1, 64), (8, 8, 129, 0, 1, 64), (4, 2, 128, 127, 1, 128), (8, 2, 65, 63, 1, 64), (8, 1, 300, 50, 1, 64),
                                                    (8, 2, 200, 77, 2, 16), (8, 2, 31, 400, 3, 64), (4, 1, 513, 1000, 2, 64)])
def test_tensor_memory_prompt_attention(nq, nkv, T, pos0, kvt, page):
    """Group sizes 1 to 8, one to several blocks of query rows and key tiles, contexts that end inside and on tiles, every page format;
    whatever lies behind the last key (here NaN) does not enter."""
    import math
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator(device=DEV).manual_seed(T + pos0)
    rand = lambda *shape: torch.randn(shape, device=DEV, generator=g)  # noqa: E731
    n = pos0 + T
    pages = (n + page - 1) // page
    table = torch.randperm(pages + 3, device=DEV, generator=g)[:pages].to(torch.int32)
    pools, scales, rows = [], [], []
    for _ in range(2):
        x = rand(pages + 3, nkv, page, 128)
        s = None
        if kvt == 1:
            q = x.half()
            d = q.double()
        else:
            top = 127 if kvt == 2 else 7
            s = (x.abs().amax(-1) / top).contiguous()
            c = (x / s[..., None]).round().clamp(-top, top)
            d = c.double() * s.double()[..., None]
            q = c.to(torch.int8) if kvt == 2 else ((c + 8).to(torch.uint8)[..., 0::2] | ((c + 8).to(torch.uint8)[..., 1::2] << 4))
        rows.append(d[table.long()].transpose(1, 2).reshape(-1, nkv, 128)[:n])
        if n % page:
            (q if s is None else s)[int(table[-1]), :, n % page:] = float("nan")
        pools.append(q.contiguous())
        scales.append(s)
    query = rand(T, nq, 128)
    got = torch.full((T, nq * 128), float("nan"), dtype=torch.float16, device=DEV)
    scratch = torch.empty(2 * nkv * 128 * ((n + 127) // 128 * 128), dtype=torch.float16, device=DEV)
    K.attn_prefill(query, pos0, table, nq, nkv, 128, kvt, page, *pools, *scales, out=got, scratch=scratch)
    hidden = torch.arange(n, device=DEV)[None] > pos0 + torch.arange(T, device=DEV)[:, None]
    for h in range(nq):
        score = query[:, h].double() @ rows[0][:, h * nkv // nq].T / math.sqrt(128)
        p = score.masked_fill(hidden, -math.inf).softmax(-1)
        v = rows[1][:, h * nkv // nq]
        # f16 queries and rows move a score by at most 3 * 2^-11 of the sum of its products' magnitudes, f16 probabilities a weight by 2^-11
        moved = (query[:, h].double().abs() @ rows[0][:, h * nkv // nq].abs().T / math.sqrt(128) * 3 * 2.0 ** -11).amax(-1, keepdim=True)
        bound = (2 * moved + 2.0 ** -10) * (p @ v.abs()) + 2.0 ** -10 * (p @ v).abs() + 1e-6
        assert ((got[:, K.paired_k_index(nq * 128, DEV)].double()[:, h * 128:(h + 1) * 128] - p @ v).abs() <= bound).all(), h


@pytest.mark.parametrize("ty", [TQ2_0_G128, Q1_0_G128])
@pytest.mark.parametrize("rows,cols,T,split", [(1, 128, 1, 0), (128, 128, 16, 1), (130, 384, 17, 2), (144, 640, 33, 3), (272, 1152, 64, 8), (2560, 512, 9, 1), (20000, 256, 40, 2)])
def test_batch_gemm_through_tensor_memory(ty, rows, cols, T, split):
    """One block of inputs and fewer blocks than CTAs in a cluster, remainders of rows (128 per tile), of blocks (four per copy, six slots)
    and of tokens (16, 32, 64), shares of the tokens that do not come out even, several tiles per cluster."""
    from oxibonsai_b200.ops import cuda_ops as K
    raw, dense = _random_quant(ty, rows, cols, rows + T)
    w = K.PlanarWeight(rows, cols, torch.device(DEV))
    w.fill_from_gguf(torch.from_numpy(np.array(raw, copy=True)).to(DEV), ty, cols, 0, rows)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn((T, cols), device=DEV, generator=g).half()
    res = torch.randn((T, rows), device=DEV, generator=g)
    paired = torch.empty_like(x)
    paired[:, K.paired_k_index(cols, DEV)] = x
    dense = dense.to(DEV).double()
    want, terms = x.double() @ dense.T, x.double().abs() @ dense.abs().T
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    bound = 2.0 ** -23 * (cols + 16) * (terms + res.abs().double())      # products are exact in f32, sums may drop a last place each
    a = K.bitgemm_batch(w, paired, 0, status=status, split=split)
    b = K.bitgemm_batch(w, paired, 1, residual=res, status=status, split=split)
    assert ((a.double() - want).abs() <= bound).all() and ((b.double() - want - res.double()).abs() <= bound).all()
    assert torch.equal(a, K.bitgemm_batch(w, paired, 0, split=split))
    if rows % 2 == 0:
        gate, up = want[:, 0::2], want[:, 1::2]
        act = torch.nn.functional.silu(gate) * up
        wide = torch.zeros((T, (rows // 2 + 15) // 16 * 16), dtype=torch.float16, device=DEV)
        K.bitgemm_batch(w, paired, 2, out=wide, status=status, split=split)
        got = wide[:, K.paired_k_index(wide.shape[1], DEV)][:, :rows // 2].double()
        slack = 1.1 * bound[:, 0::2] * up.abs() + gate.abs() * bound[:, 1::2] + (2.0 ** -11 + 2.0 ** -20) * act.abs() + 2.0 ** -24
        assert ((got - act).abs() <= slack).all()
    assert status.item() == 0


@pytest.mark.parametrize("T", [1, 5, 12, 33, 64])
@pytest.mark.parametrize("split", [3, 5, 7, 8])
def test_batch_gemm_shares_of_tokens(T, split):
    """Groups of four tokens handed out over the CTAs of a cluster: CTAs without tokens, with fewer than four, unequal shares of blocks, a last
    tile of fewer rows, one tile and several per cluster (148 / 3 clusters at most)."""
    from oxibonsai_b200.ops import cuda_ops as K
    for rows, cols in ((200, 1152), (64 * 128 + 6, 1152)):
        raw, dense = _random_quant(TQ2_0_G128, rows, cols, rows + T)
        w = K.PlanarWeight(rows, cols, torch.device(DEV))
        w.fill_from_gguf(torch.from_numpy(np.array(raw, copy=True)).to(DEV), TQ2_0_G128, cols, 0, rows)
        g = torch.Generator(device=DEV).manual_seed(T + split)
        x = torch.randn((T, cols), device=DEV, generator=g).half()
        res = torch.randn((T, rows), device=DEV, generator=g)
        paired = torch.empty_like(x)
        paired[:, K.paired_k_index(cols, DEV)] = x
        dense = dense.to(DEV).double()
        want, terms = x.double() @ dense.T + res.double(), x.double().abs() @ dense.abs().T + res.abs().double()
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        got = K.bitgemm_batch(w, paired, 1, residual=res, status=status, split=split)
        assert ((got.double() - want).abs() <= 2.0 ** -23 * (cols + 16) * terms).all()      # products are exact in f32, sums may drop a last place each
        assert status.item() == 0


def _row_scale(x, threads):
    """1 / rms of every row of x with the squares added in the order that the results depend on: thread t of `threads` adds groups t, t + threads, ..
    of four neighbouring inputs, then warps by halves, then the warps' sums by halves.  One rounding to 32 bits per step."""
    f = np.float32
    T, k = x.shape
    step = -(-k // (4 * threads)) * 4 * threads
    v = np.zeros((T, step), dtype=np.float64)
    v[:, :k] = x
    v = v.reshape(T, -1, threads, 4)
    acc = np.zeros((T, threads), dtype=f)
    for i in range(v.shape[1]):
        y = f(v[:, i, :, 1] ** 2)
        for e in (0, 2, 3):
            y = f(v[:, i, :, e] ** 2 + y.astype(np.float64))
        acc = acc + y
    def halves(a):
        while a.shape[-1] > 1:
            n = a.shape[-1] // 2
            a = a[..., :n] + a[..., n:]
        return a[..., 0]
    warps = np.zeros((T, 32), dtype=f)
    warps[:, :threads // 32] = halves(acc.reshape(T, threads // 32, 32))
    return f(1) / np.sqrt(halves(warps) / f(k) + f(1e-6))


@pytest.mark.parametrize("cols", [128, 1920, 2048, 2560, 4096, 12288, 33024])
@pytest.mark.parametrize("T", [1, 128, 129])
def test_row_norms_add_their_squares_in_a_fixed_order(cols, T):
    """f16 rows that feed the products: their bits hang on the order of the sum, whatever the block and the width of its loads."""
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator().manual_seed(cols + T)
    x = torch.randn((T, cols), generator=g) * torch.randn((T, 1), generator=g).exp()
    w = torch.randn(cols, generator=g)
    def want(threads):
        return x * (w * torch.from_numpy(_row_scale(x.numpy(), threads))[:, None])
    few = 1024 if cols >= 4096 else (512 if cols >= 2048 else 256)
    rows = want(few if T <= 128 else 256).half()
    perm, hmma = K.paired_k_index(cols, DEV), K.hmma_k_index(cols)
    assert torch.equal(K.norm_to_f16_paired(x.to(DEV), w.to(DEV), 1e-6)[:, perm].cpu(), rows)
    assert torch.equal(K.norm_to_f16_paired(x.to(DEV), w.to(DEV), 1e-6, natural=True).cpu(), rows)
    assert torch.equal(K.norm_to_f16_hmma(x.to(DEV), w.to(DEV), 1e-6).cpu()[:, hmma], want(few).half())
    # rows off 16-byte boundaries: scalar loads, blocks of the full width
    wide = torch.zeros((T, cols + 1), device=DEV)
    wide[:, 1:] = x.to(DEV)
    ref = x.double() * w.double() / (x.double().square().mean(-1, keepdim=True) + 1e-6).sqrt()
    bound = 2.0 ** -11 * ref.abs() + cols * 2.0 ** -24 * ref.abs() + 2.0 ** -24
    for got in (K.norm_to_f16_paired(wide[:, 1:], w.to(DEV), 1e-6)[:, perm].cpu(), K.norm_to_f16_hmma(wide[:, 1:], w.to(DEV), 1e-6).cpu()[:, hmma]):
        assert ((got.double() - ref).abs() <= bound).all()


@pytest.fixture(scope="module")
def wide_head_gguf(tmp_path_factory):
    from oxibonsai_b200.core import Qwen3Config, write_synthetic_gguf
    p = tmp_path_factory.mktemp("gguf") / "wide_head.gguf"
    write_synthetic_gguf(str(p), Qwen3Config(hidden=512, inter=1024, layers=2, heads=4, kv_heads=2, head_dim=128, vocab=1000, context=1024, name="wide"), seed=3)
    return str(p)


@pytest.mark.parametrize("T", [16, 32, 33, 64, 65, 256])
def test_short_prompts_over_int4_pages_keep_their_kernels(T, wide_head_gguf):
    """The cache rows that a prompt leaves behind are, bit for bit, those of the former kernels one by one: another order of their sums would flip
    codes.  Above 64 tokens that includes products over expanded weights."""
    from oxibonsai_b200.ops import cuda_ops as K
    from oxibonsai_b200.runtime import EngineBuilder
    eng = EngineBuilder().model_path(wide_head_gguf).max_seq_len(320).max_batch(2).kv_cache("q4").build()
    r, cfg = eng.runner, eng.runner.cfg
    prompt = torch.randint(0, cfg.vocab, (T,), generator=torch.Generator().manual_seed(T)).tolist()
    eng.begin_sequence(prompt, T + 1, 0)
    eng.prefill(prompt, 0, 0)
    torch.cuda.synchronize()
    got = [t.clone() for t in (eng.kv.k, eng.kv.v, eng.kv.k_scale, eng.kv.v_scale)]
    for t in (eng.kv.k, eng.kv.v, eng.kv.k_scale, eng.kv.v_scale):
        t.zero_()
    nq, nkv, eps = cfg.heads, cfg.kv_heads, cfg.eps
    table = r.block_table[:1].contiguous()
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    h = torch.index_select(r.w.embd, 0, torch.tensor(prompt, device=DEV)).float()
    splits = max(1, min(16, 4 * 148 // (nkv * T)))
    splits = 1 << (splits.bit_length() - 1)
    to_f16, gemm = (K.norm_to_f16_hmma, K.bitgemm_hmma) if T <= 32 else (K.norm_to_f16_paired, K.bitgemm_prefill)
    for l, lw in enumerate(r.w.layers):
        pools = (eng.kv.k[l], eng.kv.v[l], eng.kv.k_scale[l], eng.kv.v_scale[l])
        qkv = gemm(lw.qkv, to_f16(h, lw.attn_norm, eps))
        q = torch.empty((T, nq, 128), device=DEV)
        K.qknorm_rope_kvstore(qkv, lw.q_norm, lw.k_norm, eps, r.rope_cos, r.rope_sin, pos, table.expand(T, -1).contiguous(), q, nq, nkv, 128, 3, eng.kv.page_size, *pools)
        if T <= 32:
            K.lib().bonsai_attn_decode_force_cuda_cores(1)
            try:
                a = K.attn_decode(q, pos, table.expand(T, -1).contiguous(), nq, nkv, 128, 3, eng.kv.page_size, *pools, nsplit=splits)
            finally:
                K.lib().bonsai_attn_decode_force_cuda_cores(0)
            a = to_f16(a.view(T, -1))
        else:
            a = K.attn_prefill(q, 0, table[0], nq, nkv, 128, 3, eng.kv.page_size, *pools)
        h = gemm(lw.o, a, epi=1, residual=h)
        h = gemm(lw.down, gemm(lw.gate_up, to_f16(h, lw.ffn_norm, eps), epi=2), epi=1, residual=h)
    for a, b in zip(got, (eng.kv.k, eng.kv.v, eng.kv.k_scale, eng.kv.v_scale)):
        assert torch.equal(a, b)
    assert torch.equal(r._pf["h"][:T], h)


@pytest.mark.parametrize("scale", [6e-8, 3e-5, 511.5, 512.0, 60000.0])
def test_batch_gemm_takes_every_scale_of_the_format(scale):
    """Group scales are f16: the smallest subnormal to the largest, one row with it among ordinary ones and all rows."""
    from oxibonsai_b200.ops import cuda_ops as K
    g = torch.Generator(device=DEV).manual_seed(1)
    raw, _ = _random_quant(TQ2_0_G128, 200, 512, 3)
    w = K.PlanarWeight(200, 512, torch.device(DEV)).fill_from_gguf(torch.from_numpy(np.array(raw, copy=True)).to(DEV), TQ2_0_G128, 512, 0, 200)
    x = (torch.randn((20, 512), device=DEV, generator=g) * 1e-3).half()
    paired = torch.empty_like(x)
    paired[:, K.paired_k_index(512, DEV)] = x
    w.scales.fill_(1.0)
    signs = K.expand_rows(w)[:, K.paired_k_index(512, DEV)].double()      # -1, 0, +1
    assert signs.abs().max() == 1.0
    for rows in (slice(77, 78), slice(0, 200)):
        w.scales.fill_(0.02)
        w.scales[rows] = scale
        dense = signs * w.scales.double().repeat_interleave(128, 1)
        assert torch.equal(K.expand_rows(w)[:, K.paired_k_index(512, DEV)].double(), dense)
        want, terms = x.double() @ dense.T, x.double().abs() @ dense.abs().T
        assert ((K.bitgemm_batch(w, paired).double() - want).abs() <= 2.0 ** -23 * 528 * terms).all()
