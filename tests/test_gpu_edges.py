"""Kernels and dispatches at the sizes where they can go wrong: edges of tiles, remainders, the
smallest and the largest that a variant takes."""
import math

import pytest
import torch

from nimbus_infer_rs_b200.csrc import ops as ops_mod
from nimbus_infer_rs_b200.engine.batch import build_layout
from test_gpu_kernels import _attention_ref, _paged_cache

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    return ops_mod.backend()


@pytest.fixture(autouse=True)
def own_random_numbers():
    """What is drawn here moves no other test's numbers."""
    with torch.random.fork_rng():
        yield


@pytest.mark.parametrize("width, pair", [(96, 1), (128, 1), (192, 1), (256, 1), (96, 0), (128, 0)])
@pytest.mark.parametrize("M, N, K", [(129, 260, 8), (257, 1600, 136), (511, 52, 640), (2900, 516, 72), (5000, 2052, 72),
                                     (5000, 2052, 648)])
def test_tiles_of_every_width_with_32_bit_results(ops, width, pair, M, N, K):
    """One tile and several a CTA, rows and columns that end inside a 32 x 32 box, K shorter and longer
    than the ring; the residual added in place.  Sums of K products in fp32: 3e-6 of the largest for
    64 of them."""
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) / math.sqrt(K)).bfloat16()
    bias, res = torch.randn(N, device=DEV), torch.randn(M, N, device=DEV)
    ref = x.double() @ w.double().t() + bias.double()
    tol = 3e-6 * float(ref.abs().max()) * math.sqrt(max(K, 64) / 64)
    ops.lib.nb_gemm_tcgen05_force(width, pair)
    try:
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.linear(x, w, bias, out)
        stream = res.clone()
        ops.linear(x, w, bias, stream, 0, stream)
        ops.check_device_errors()
    finally:
        ops.lib.nb_gemm_tcgen05_force(0, 0)
    assert (out.double() - ref).abs().max() <= tol
    want = ref + res.double()
    assert (stream.double() - want).abs().max() <= tol + 1e-6 * float(want.abs().max())


def test_a_product_without_a_kernel_of_the_width_that_is_set_is_refused(ops):
    """By the result's type, by its rows (up to 128 take tiles of their own), by rows that TMA cannot store."""
    x, w = (torch.randn(n, 64, device=DEV).bfloat16() for n in (300, 260))
    for (width, pair), rows, columns, dtype in (((96, 0), 300, 260, torch.bfloat16), ((192, 0), 300, 260, torch.float32),
                                                ((128, 0), 100, 260, torch.float32), ((128, 0), 300, 257, torch.float32)):
        out = torch.zeros(rows, columns, device=DEV, dtype=dtype)
        assert ops.lib.nb_gemm_tcgen05_force(width, pair) == 0
        try:
            with pytest.raises(ops_mod.KernelError):
                ops._call("nb_gemm_tcgen05", x.data_ptr(), w.data_ptr(), 0, 0, out.data_ptr(), int(dtype == torch.bfloat16),
                          rows, columns, 64, 0, torch.cuda.current_stream().cuda_stream)
        finally:
            ops.lib.nb_gemm_tcgen05_force(0, 0)
        assert (out == 0).all()


@pytest.mark.parametrize("columns", [96, 128])
@pytest.mark.parametrize("M, N, K", [(65, 95, 64), (128, 97, 520), (129, 193, 1032), (70, 300, 4104)])
def test_32_bit_products_in_tiles_of_either_width(ops, columns, M, N, K):
    """Tiles of 96 and 128 columns, K of up to and beyond the blocks whose small terms share an
    accumulator, rows that a warp, four warps and more than those hold while they are split; a row
    without pieces.  Within half of what one sequence of multiply-adds could be off."""
    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device=DEV)
    w = torch.randn(N, K, device=DEV) / math.sqrt(K)
    x[3, K - 1] = 2.0 ** 60
    ref = x.double() @ w.double().t()
    was, ops.use_f32_tc = ops.use_f32_tc, 2
    ops.lib.nb_gemm_f32_tc_force(columns)
    try:
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.linear(x, w, None, out)
        ops.check_device_errors()
    finally:
        ops.use_f32_tc = was
        ops.lib.nb_gemm_f32_tc_force(0)
    err = (out.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err.max()) <= 2.0 ** -24 * max(4.0, 0.5 * math.sqrt(K))


@pytest.mark.parametrize("H, Hk, hd, window", [(3, 3, 64, 0), (4, 2, 64, 65), (2, 1, 128, 0)])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_32_bit_prompt_attention_at_the_edges_of_its_tiles(ops, dtype, H, Hk, hd, window, shift):
    """Rows and keys around a tile's 64, chunks behind a cached context, more tiles than SMs; with
    ``shift`` the rows' numbers cannot be taken four at a time.  A bfloat16 cache through the same
    kernel (its own entry point)."""
    lens = [64, 65, 1, 130, 63, 2000]
    new = [64, 65, 1, 2, 63, 1999]
    kv, dk, dv = _paged_cache(len(lens), lens, Hk, hd, dtype, seed=hd + H)
    lay = build_layout([(s + 1, [0] * n, []) for s, n in enumerate(new)], [l - n for l, n in zip(lens, new)], DEV)
    torch.manual_seed(9)
    q = torch.randn(lay.n_rows, H * hd + shift, device=DEV).to(dtype)
    out = torch.full((lay.n_rows, H * hd), 7.0, device=DEV)
    scale = 0.37 / math.sqrt(hd)
    rc = ops.lib.nb_attention_prefill_f32(
        q.data_ptr(), 0 if dtype == torch.float32 else 1, q.shape[1], shift, lay.cu_rows.data_ptr(), lay.seq_slot.data_ptr(),
        lay.seq_pos0.data_ptr(), kv.k.data_ptr(), kv.v.data_ptr(), kv.block_table.data_ptr(), kv.block_table.shape[1], 64,
        H, Hk, hd, out.data_ptr(), 0, H * hd, scale, window, len(new), max(new), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    r = 0
    for s, n in enumerate(new):
        for i in range(n) if n < 200 else (0, 62, 63, 64, n // 2, n - 1):
            ref = _attention_ref(q[r + i, shift:].view(H, hd).cpu(), dk[s], dv[s], lens[s] - n + i, scale, H // Hk, window)
            got = out[r + i].view(H, hd).double().cpu()
            assert (got - ref).abs().max() <= 2e-5 * max(1.0, float(ref.abs().max())), (s, i)
        r += n


def test_a_session_that_runs_ahead_of_the_device(tmp_path):
    """Tokens from the host for many steps with nothing read in between, steps without tokens among
    them, and a step that is refused: the logits of plain steps.  More tokens than one launch carries."""
    ops, many = ops_mod.backend(), torch.zeros(1923, dtype=torch.int32, device=DEV)
    ops.set_tokens(many, torch.arange(7, 1930, dtype=torch.int32))
    assert many.tolist() == list(range(7, 1930))
    from nimbus_infer_rs_b200 import Engine
    from nimbus_infer_rs_b200.engine.decode import DecodeSession
    from tiny_configs import make_model
    engine = Engine.load(make_model(tmp_path, "A"), dtype="float32", device=DEV, cache_tokens=1024)
    prompts, fed = [[5, 17, 3], [7] * 9], [[k * 7 % 90 + 1, k * 5 % 90 + 2] for k in range(11)]
    plain = [engine.alloc_slot() for _ in prompts]
    engine.step([(s, p) for s, p in zip(plain, prompts)])
    want = None
    for t in fed:
        want = engine.step([(s, [x]) for s, x in zip(plain, t)])
    for _ in range(2):                           # the second session finds the first one's recording
        slots = [engine.alloc_slot() for _ in prompts]
        engine.step([(s, p) for s, p in zip(slots, prompts)])
        session = DecodeSession(engine, slots, fed[0])
        session.step()                           # the first tokens lie on the device
        for t in fed[1:]:
            session.step(t)
        with pytest.raises(ValueError):
            session.step([1, 2, 3])              # three tokens for two rows
        assert session.read_tokens() == session.logits.argmax(1).tolist()
        torch.testing.assert_close(session.logits, want, rtol=0, atol=2e-5 * float(want.abs().max()))
        session.step()                           # what was selected, as it lies on the device
        session.step(fed[0])
        session.close()
        for s in slots:
            engine.free_slot(s)


@pytest.mark.parametrize("rows, H, Hk", [(50, 12, 12), (74, 12, 12), (64, 25, 25), (60, 24, 12)])
@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("append", [False, True])
def test_decode_attention_of_large_batches_over_heads_of_64(ops, rows, H, Hk, window, append):
    """Whole sequences in more than four CTAs an SM (two warps, 32 keys each), below and beyond what is on
    the GPU at once: lengths around a page's end and of one to six pages, a padding row, NaN in every row of
    a page that holds no key, the step's own keys and values from its rows or from the cache.  Off by at
    most the rounding of probabilities and results to 8 bits: 2^-9 of the largest value and of the
    result."""
    hd, dtype = 64, torch.bfloat16
    lens = [(1, 63, 64, 65, 129, 200, 333, 128)[i % 8] for i in range(rows)]
    kv, dk, dv = _paged_cache(rows, lens, Hk, hd, dtype, seed=rows + H, stale_nan=True)
    lay = build_layout([(s + 1, [0], []) for s in range(rows)], [n - 1 for n in lens], DEV)
    lay.row_slot[2] = -1
    torch.manual_seed(8)
    qkv = torch.randn(rows, (H + 2 * Hk) * hd, device=DEV).to(dtype)
    pages = kv.block_table[torch.arange(1, rows + 1, device=DEV), torch.tensor([(n - 1) // 64 for n in lens], device=DEV)].long()
    at = torch.tensor([(n - 1) % 64 for n in lens], device=DEV)
    if append:
        own = [t.view(rows, Hk, hd) for t in (qkv[:, H * hd:(H + Hk) * hd], qkv[:, (H + Hk) * hd:])]
        for dense, mine, plane in zip((dk, dv), own, (kv.k, kv.v)):
            plane[pages, :, at] = float("nan")
            for s in range(rows):
                dense[s][-1] = mine[s].cpu()
    out = torch.full((rows, H * hd), 7.0, device=DEV, dtype=dtype)
    scale = 0.5 / math.sqrt(hd)
    ops.attention(qkv, 0, lay, kv, H, out, scale, window, append=(H * hd, (H + Hk) * hd) if append else None)
    for s, n in enumerate(lens):
        if s == 2:
            assert (out[s] == 0).all()
            continue
        ref = _attention_ref(qkv[s, :H * hd].view(H, hd).cpu(), dk[s], dv[s], n - 1, scale, H // Hk, window)
        err = (out[s].view(H, hd).double().cpu() - ref).abs().max()
        assert err <= 2.0 ** -9 * float(dv[s].double().abs().max() + ref.abs().max()) + 1e-4, s
    if append:      # the cache holds them now; the padding row has written nothing
        live = [s for s in range(rows) if s != 2]
        for mine, plane in zip(own, (kv.k, kv.v)):
            assert torch.equal(plane[pages, :, at][live], mine[live]) and plane[pages, :, at][2].isnan().all()


@pytest.mark.parametrize("rows, H, Hk, longest", [(2, 2, 2, 1530), (3, 16, 4, 1100), (40, 16, 4, 330), (9, 16, 2, 700),
                                                  (5, 8, 1, 961), (12, 12, 6, 577)])
def test_decode_attention_of_small_batches_over_heads_of_64(ops, rows, H, Hk, longest):
    """Splits by eight warps (shared key heads in up to a CTA an SM; more than two pages a split) and by
    four, over one long sequence among short ones, an odd number of pages, and a split whose pages lie beyond
    most sequences.  Bound as above."""
    hd, dtype = 64, torch.bfloat16
    lens = [longest if s == rows // 2 else (1, 65, 130, 64, 257)[s % 5] for s in range(rows)]
    kv, dk, dv = _paged_cache(rows, lens, Hk, hd, dtype, seed=rows + H, stale_nan=True)
    lay = build_layout([(s + 1, [0], []) for s in range(rows)], [n - 1 for n in lens], DEV)
    lay.max_kv_len = longest
    torch.manual_seed(8)
    q = torch.randn(rows, H * hd, device=DEV).to(dtype)
    out = torch.full((rows, H * hd), 7.0, device=DEV, dtype=dtype)
    scale = 0.5 / math.sqrt(hd)
    ops.attention(q, 0, lay, kv, H, out, scale)
    for s, n in enumerate(lens):
        ref = _attention_ref(q[s].view(H, hd).cpu(), dk[s], dv[s], n - 1, scale, H // Hk)
        err = (out[s].view(H, hd).double().cpu() - ref).abs().max()
        assert err <= 2.0 ** -9 * float(dv[s].double().abs().max() + ref.abs().max()) + 1e-4, s
