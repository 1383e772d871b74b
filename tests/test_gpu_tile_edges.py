"""Edges of the kernels' tiles and of their dispatch against the CPU oracle: the INT4 GEMM's row tiles,
uneven widths and scales on either side of its two ways to dequantize; the decode and verify kernels at
uneven widths and expert counts, with tied experts and with every row on the same experts; the row kernels
at the widths where they change form and with rows that are not 16-byte aligned."""
import numpy as np
import pytest

from ane_fieldfare_b200 import gturbo, synth, workload
from conftest import LAYER_ELEMENTWISE_TOL, assert_layer_close, oracle_layer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def context(L, rows):
    from ane_fieldfare_b200 import hotpath as hp
    ctx = hp.HotpathContext(layers=1, experts=L.experts, d=L.d, f=L.f, sharedF=L.sharedF, topK=L.topK, maxTokens=rows)
    workload.load_layer(ctx, 0, L)
    return hp, ctx


@pytest.mark.parametrize("scales", ["small", "mixed"])
@pytest.mark.parametrize("d,fs", [(64, 64), (192, 320), (2816, 704), (6400, 128)])
@pytest.mark.parametrize("rows", [17, 33, 64, 65, 97, 192, 193, 385])
def test_int4_gemm_shapes_and_scales(oracle, scales, d, fs, rows):
    L = workload.make_layer(0x71, 0, experts=8, d=d, f=64, sharedF=fs, topK=2)
    if scales == "mixed":
        # rows of 32-fold scales (above 2^-5), of zero and of subnormal ones beside the ordinary
        L.sharedBlob = L.sharedBlob.copy()
        for name in ("gate", "up"):
            _, s, b = gturbo.sub_tensor(L.sharedBlob, L.sharedLayout, name)
            s, b = s.reshape(fs, d // 64), b.reshape(fs, d // 64)
            s[5::40] += np.uint16(5 << 7)
            b[5::40] += np.uint16(5 << 7)
            s[9] = 0
            s[17] = np.uint16(0x0035)
    hp, ctx = context(L, 400)
    try:
        x = workload.make_tokens(0x72, f"edges{rows}", rows, d)
        y = torch.zeros((rows, d), dtype=torch.bfloat16, device=ctx.device)
        hp.PrefillSharedExpert(ctx).encodeBlock(None, 0, hp.bf16_tensor(x, ctx.device), y, rows)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want = oracle.shared_ffn(oracle_layer(oracle, L), x, bf16_weights=True)
        # (outputs here reach the thousands and cancel: the norm of the error, well inside the bound)
        rel_l2, _, _ = assert_layer_close(hp.bf16_numpy(y), want, oracle, f"int4 gemm {d}x{fs} rows={rows} {scales}")
        assert rel_l2 < 2e-3
    finally:
        ctx.close()


@pytest.mark.parametrize("experts,d,f,fs,k", [(5, 128, 64, 64, 1), (9, 192, 128, 320, 3), (130, 448, 192, 64, 8),
                                              (16, 2816, 704, 0, 8)])
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 16, 40])
def test_block_shapes(oracle, experts, d, f, fs, k, rows):
    L = workload.make_layer(0x73, 0, experts=experts, d=d, f=f, sharedF=fs, topK=k)
    L.routerW[3] = L.routerW[1]  # tied logits: the lower id comes first
    hp, ctx = context(L, 40)
    try:
        ld = oracle_layer(oracle, L)
        x = workload.make_tokens(0x74, f"block{rows}", rows, d)
        if rows == 5:
            x[:] = x[0]  # every row on the same experts
        ids = torch.zeros((rows, k), dtype=torch.int32, device=ctx.device)
        y = ctx.moeLayer(0, hp.bf16_tensor(x, ctx.device), ids=ids)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want, _, ref_ids, _ = oracle.moe_layer(ld, x, oracle.MODE_PARTIALS | (oracle.MODE_BF16_WEIGHTS if rows > 16 else 0))
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ref_ids)
        assert_layer_close(hp.bf16_numpy(y), want, oracle, f"block {experts}x{d}x{f}+{fs} rows={rows}",
                           elementwise_tol=LAYER_ELEMENTWISE_TOL)
        if rows == 5:
            assert torch.equal(y, y[:1].expand(5, d))
    finally:
        ctx.close()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("d", [64, 4096, 4160, 16384, 16448])
def test_row_kernels(oracle, d, shift):
    """`shift`: rows start that many elements behind an aligned address."""
    from ane_fieldfare_b200 import hotpath as hp
    rows, eps = 3, 1e-6
    ctx = hp.HotpathContext(layers=1, experts=8, d=d, f=64, sharedF=0, topK=2, maxTokens=4)
    try:
        def dev(bits):
            bits = np.asarray(bits, dtype=np.uint16)
            t = torch.empty(bits.size + 8, dtype=torch.bfloat16, device=ctx.device)
            v = t[shift:shift + bits.size].view(bits.shape)
            v.copy_(hp.bf16_tensor(bits, ctx.device))
            return v

        mk = lambda seed, shape, a: synth.bf16_bits(synth.uniform(seed, int(np.prod(shape)), -a, a)).reshape(shape)
        hidden, attn, h2, h1 = (mk(80 + i, (rows, d), 2.0) for i in range(4))
        w = [synth.bf16_bits(synth.uniform(90 + i, d, 0.5, 1.5)) for i in range(5)]
        hd, dense, routed, router, tail = dev(hidden), dev(h1), dev(h1), dev(h1), dev(hidden)
        glue = hp.PrefillLayerGlue(ctx)
        glue.encodePostAttnSetupBlock(None, hd, dev(attn), dev(w[0]), dev(w[1]), dev(w[2]), eps, dense, routed, router)
        glue.encodeLayerTailBlock(None, dev(h2), dev(h1), tail, dev(w[3]), dev(w[4]), eps, 0.7071)
        norm = ctx.rmsnorm(dev(hidden), dev(w[0]), eps, dev(h1))
        torch.cuda.synchronize()
        want = [*oracle.post_attn_setup(hidden, attn, w[0], w[1], w[2], eps),
                oracle.layer_tail(h2, h1, hidden, w[3], w[4], eps, 0.7071), oracle.rmsnorm_bf16(hidden, w[0], eps, rows, d)]
        for got, ref in zip((hd, dense, routed, router, tail, norm), want):
            g, r = oracle.bf16_to_float(hp.bf16_numpy(got)), oracle.bf16_to_float(ref)
            assert np.all(np.abs(g - r) <= np.maximum(np.abs(r), 4.0) * 2.0 ** -7 * 1.01)
            assert np.mean(g != r) < 1e-2
    finally:
        ctx.close()


@pytest.mark.parametrize("rows", [40, 700])
def test_gemms_repeat_bit_for_bit(rows):
    """The CTA pairs' hand-overs: the same rows again and again beside other traffic on the chip give the same bits."""
    from test_gpu_router_int8 import int8_projection
    L = workload.make_layer(0x75, 0, experts=32, d=1088, f=320, sharedF=704, topK=8)
    hp, ctx = context(L, rows)
    int8 = hp.HotpathContext(layers=1, experts=8, d=1088, f=64, sharedF=704, topK=8, maxTokens=rows)
    try:
        int8.loadSharedInt8(0, int8_projection(1, 704, 1088, 0.02), int8_projection(2, 704, 1088, 0.02),
                            int8_projection(3, 1088, 704, 0.02))
        x = hp.bf16_tensor(workload.make_tokens(0x76, f"repeat{rows}", rows, 1088), ctx.device)
        other = torch.cuda.Stream()
        src = torch.ones(1 << 26, dtype=torch.uint8, device=ctx.device)
        dst = torch.empty_like(src)
        first = None
        for i in range(12):
            with torch.cuda.stream(other):
                for _ in range(i % 4):
                    dst.copy_(src)
            y8 = torch.empty_like(x)
            hp.PrefillSharedExpert(int8).encodeBlock(None, 0, x, y8, rows)
            out = (ctx.moeLayer(0, x), y8)
            torch.cuda.synchronize()
            first = first or out
            assert torch.equal(out[0], first[0]) and torch.equal(out[1], first[1])
        assert ctx.info().deviceErrorFlag == 0 and int8.info().deviceErrorFlag == 0
    finally:
        int8.close()
        ctx.close()


@pytest.mark.parametrize("d,f,fs,rows", [(192, 320, 64, 384), (192, 320, 64, 385), (448, 128, 0, 769), (128, 64, 320, 8000),
                                         (320, 64, 192, 8193)])
def test_int4_gemm_tile_rows(oracle, d, f, fs, rows):
    """Rows on either side of where the routed GEMMs (96 an expert) and the shared FFN's (whole waves) go over from tiles of
    128 rows to 192, with contractions that end inside a quad of steps, in its first pair or its second."""
    L = workload.make_layer(0x77, 0, experts=8, d=d, f=f, sharedF=fs, topK=2)
    hp, ctx = context(L, rows)
    try:
        ld = oracle_layer(oracle, L)
        x = workload.make_tokens(0x78, f"tiles{rows}", rows, d)
        ids = torch.zeros((rows, 2), dtype=torch.int32, device=ctx.device)
        y = ctx.moeLayer(0, hp.bf16_tensor(x, ctx.device), ids=ids)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want, _, ref_ids, _ = oracle.moe_layer(ld, x, oracle.MODE_PARTIALS | oracle.MODE_BF16_WEIGHTS)
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ref_ids)
        # the kernels and the oracle round the same sums to bf16: 2^-9 at most where they fall on other sides
        rel_l2, _, _ = assert_layer_close(hp.bf16_numpy(y), want, oracle, f"tile rows {d}x{f}+{fs} rows={rows}")
        assert rel_l2 < 2.0 ** -9
    finally:
        ctx.close()


@pytest.mark.parametrize("d,f,fs", [(3712, 64, 64), (5120, 64, 64), (9856, 64, 0), (128, 2688, 64), (128, 4096, 4096), (64, 7808, 64)])
@pytest.mark.parametrize("rows", [384, 385])
def test_int4_gemm_ring_sizes(oracle, d, f, fs, rows):
    """Contractions that give the GEMMs each number of code slots and scale buffers, with tiles of 128 rows (up to 384 rows of two
    routes to eight experts) and of 192: the oracle's rows, and the same bits beside other traffic on the chip."""
    L = workload.make_layer(0x79, 0, experts=8, d=d, f=f, sharedF=fs, topK=2)
    hp, ctx = context(L, rows)
    try:
        x = workload.make_tokens(0x7A, f"rings{rows}", rows, d)
        xd, src = hp.bf16_tensor(x, ctx.device), torch.ones(1 << 26, dtype=torch.uint8, device=ctx.device)
        ids = torch.zeros((rows, 2), dtype=torch.int32, device=ctx.device)
        other, dst, first = torch.cuda.Stream(), torch.empty_like(src), None
        for i in range(6):
            with torch.cuda.stream(other):
                for _ in range(i % 3):
                    dst.copy_(src)
            y = ctx.moeLayer(0, xd, ids=ids)
            torch.cuda.synchronize()
            first = y.clone() if first is None else first
            assert torch.equal(y, first)
        assert ctx.info().deviceErrorFlag == 0
        want, _, ref_ids, _ = oracle.moe_layer(oracle_layer(oracle, L), x, oracle.MODE_PARTIALS | oracle.MODE_BF16_WEIGHTS)
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ref_ids)
        # the kernels and the oracle round the same sums to bf16: 2^-9 at most where they fall on other sides
        rel_l2, _, _ = assert_layer_close(hp.bf16_numpy(y), want, oracle, f"rings {d}x{f}+{fs} rows={rows}")
        assert rel_l2 < 2.0 ** -9
    finally:
        ctx.close()


@pytest.mark.parametrize("top", [1, 2, 3, 8])
@pytest.mark.parametrize("rows", [70, 2368, 2369])
def test_reduce_at_every_form(oracle, top, rows):
    """Up to four CTAs an SM (2368 rows of 512 on 148) and beyond, with the partial rows streamed and not: the oracle's bits."""
    from ane_fieldfare_b200 import hotpath as hp
    d = 512
    ctx = hp.HotpathContext(layers=1, experts=8, d=d, f=64, sharedF=0, topK=top, maxTokens=rows)
    try:
        p = synth.bf16_bits(synth.uniform(1, rows * top * d, -2, 2)).reshape(rows * top, d)
        w = synth.bf16_bits(synth.uniform(2, rows * top, 0, 1)).reshape(rows, top)
        r = synth.bf16_bits(synth.uniform(3, rows * d, -1, 1)).reshape(rows, d)
        for residual in (None, r):
            y = torch.zeros((rows, d), dtype=torch.bfloat16, device=ctx.device)
            hp.PrefillMoE(ctx).encodeReduceTokenMajor(None, hp.bf16_tensor(p, ctx.device), hp.bf16_tensor(w, ctx.device), y, rows,
                                                      residual=None if residual is None else hp.bf16_tensor(residual, ctx.device))
            torch.cuda.synchronize()
            assert np.array_equal(hp.bf16_numpy(y), oracle.reduce_token_major(p, w, residual, rows, top, d))
    finally:
        ctx.close()
