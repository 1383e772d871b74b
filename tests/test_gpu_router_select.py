"""A prefill chunk's routes against the kernels that form every logit in the defined order (the same call with the
logits asked for, or blocks of 16 rows, which other tests pin against the oracle): ids and weights bit for bit, with
tied experts, all-zero, non-finite and huge rows and a bias of -inf.  A short chunk has every logit formed in one launch;
the rest goes through approximate logits on the tensor cores and exact ones of the experts that can matter, at the
edges of its token tiles (32, 64, 96 and 128 rows) and with every number of warps a row."""
import numpy as np
import pytest

from ane_fieldfare_b200 import synth, workload
from test_gpu_router_int8 import int8_router

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def load_router(ctx, form, experts, d):
    """A router with tied experts (8 to 11) and one of bias -inf."""
    bias = synth.normal(3, experts).astype(np.float32)
    bias[1] = -np.inf
    bias[8:12] = bias[8]  # (with equal weights below: exact ties)
    eff = gain = None
    if form != "bf16":
        eff = synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
        gain = synth.bf16_bits(synth.uniform(8, experts, 0.5, 1.5))
    if form == "int8":
        codes, scales, biases = int8_router(0x31, experts, d)
        for m in (codes, scales, biases):
            m[8:12] = m[8]
        ctx.loadRouterInt8(0, codes, scales, biases, effectiveScale=eff, perExpertScale=gain, logitBias=bias)
    else:
        w = synth.normal_bf16(0x32, "select.router", (experts, d), 0.02)
        w[8:12] = w[8]
        ctx.loadRouter(0, w, effectiveScale=eff, perExpertScale=gain, logitBias=bias)


def special_rows(hp, ctx, rows, d):
    """Rows d + 8 apart, zero, non-finite, huge and tiny ones among them."""
    wide = torch.zeros((rows, d + 8), dtype=torch.bfloat16, device=ctx.device)
    wide[:, :d] = hp.bf16_tensor(workload.make_tokens(0x33, f"select{rows}", rows, d), ctx.device)
    wide[1, :d] = 0
    wide[2, 5] = float("nan")
    wide[3, 6] = float("inf")
    wide[4, :d] *= 1e30
    wide[5, :d] *= 1e-30
    wide[6, 7] = 3e4
    return wide


@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("experts,d,k", [(16, 128, 8), (128, 2816, 8), (256, 448, 3), (130, 2496, 8)])
@pytest.mark.parametrize("rows", [17, 32, 129, 700])
def test_selected_routes_equal_the_exact_ones(form, experts, d, k, rows):
    from ane_fieldfare_b200 import hotpath as hp
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=700)
    try:
        bias = synth.normal(3, experts).astype(np.float32)
        bias[1] = -np.inf
        bias[8:12] = bias[8]  # (with equal weights below: exact ties)
        eff = gain = None
        if form != "bf16":
            eff = synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
            gain = synth.bf16_bits(synth.uniform(8, experts, 0.5, 1.5))
        if form == "int8":
            codes, scales, biases = int8_router(0x31, experts, d)
            for m in (codes, scales, biases):
                m[8:12] = m[8]
            ctx.loadRouterInt8(0, codes, scales, biases, effectiveScale=eff, perExpertScale=gain, logitBias=bias)
        else:
            w = synth.normal_bf16(0x32, "select.router", (experts, d), 0.02)
            w[8:12] = w[8]
            ctx.loadRouter(0, w, effectiveScale=eff, perExpertScale=gain, logitBias=bias)
        x = hp.bf16_tensor(workload.make_tokens(0x33, f"select{rows}", rows, d), ctx.device)
        wide = torch.zeros((rows, d + 8), dtype=torch.bfloat16, device=ctx.device)
        wide[:, :d] = x
        wide[1, :d] = 0
        wide[2, 5] = float("nan")
        wide[3, 6] = float("inf")
        wide[4, :d] *= 1e30
        wide[5, :d] *= 1e-30
        wide[6, 7] = 3e4
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(2)]
        weights = [torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device) for _ in range(2)]
        logits = torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)
        router = hp.PrefillRouter(ctx)
        router.encodeGemma4Block(None, 0, wide, got[0], weights[0], rows, d + 8, outLogits=logits)
        router.encodeGemma4Block(None, 0, wide, got[1], weights[1], rows, d + 8)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        assert torch.equal(got[0], got[1])
        assert torch.equal(weights[0].view(torch.int16), weights[1].view(torch.int16))
    finally:
        ctx.close()

@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("experts,d,k", [(16, 128, 8), (128, 2816, 8), (256, 448, 3), (130, 2496, 8)])
@pytest.mark.parametrize("rows", [161, 192, 300])
def test_selected_routes_behind_approximate_logits(form, experts, d, k, rows):
    """The same where the two launches run with eight warps a row."""
    test_selected_routes_equal_the_exact_ones(form, experts, d, k, rows)


@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("weights_times", [1.0, 2.0 ** -80, 2.0 ** 60])
def test_selected_routes_of_tiny_and_huge_rows(form, weights_times):
    """Without a bias, which would decide the ranks of such rows: rows whose squares vanish or overflow in fp32, whose
    products underflow, subnormal ones, and rows that mix the scales."""
    from ane_fieldfare_b200 import hotpath as hp
    experts, d, k, per = 128, 2816, 8, 12
    scales = [2.0 ** e for e in (-130, -126, -110, -90, -78, -75, -60, -50, -49, 0, 60, 64, 100, 118)]
    rows = per * (len(scales) + 1)
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)

    def times(bits):  # by a power of two
        return synth.bf16_bits(synth.bf16_to_float(bits) * np.float32(weights_times)).reshape(bits.shape)

    try:
        eff = None if form == "bf16" else synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
        if form == "int8":
            codes, s, b = int8_router(0x35, experts, d)
            ctx.loadRouterInt8(0, codes, times(s), times(b), effectiveScale=eff)
        else:
            ctx.loadRouter(0, times(synth.normal_bf16(0x36, "tiny.router", (experts, d), 0.02)), effectiveScale=eff)
        x = synth.bf16_to_float(workload.make_tokens(0x37, "tiny", rows, d)).reshape(rows, d)
        for i, v in enumerate(scales):
            x[i * per:(i + 1) * per] *= np.float32(v)
        mixed = x[len(scales) * per:]
        mixed *= np.exp2(np.rint(synth.uniform(9, mixed.size, -120, 20))).astype(np.float32).reshape(mixed.shape)
        xd = hp.bf16_tensor(synth.bf16_bits(x), ctx.device)
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(2)]
        weights = [torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device) for _ in range(2)]
        logits = torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)
        router = hp.PrefillRouter(ctx)
        router.encodeGemma4Block(None, 0, xd, got[0], weights[0], rows, outLogits=logits)
        router.encodeGemma4Block(None, 0, xd, got[1], weights[1], rows)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        wrong = (got[0] != got[1]).any(dim=1).nonzero().flatten().tolist()
        assert not wrong, wrong
        assert torch.equal(weights[0].view(torch.int16), weights[1].view(torch.int16))
    finally:
        ctx.close()


@pytest.mark.parametrize("form", ["bf16", "int8"])
@pytest.mark.parametrize("rows", [443, 445, 1184, 1777, 4000])
def test_selected_routes_at_every_number_of_warps(form, rows):
    """Rows on either side of where a row gets fewer warps (148 SMs: 444, 888, 1776 rows; INT8 592, 1184)."""
    from ane_fieldfare_b200 import hotpath as hp
    experts, d, k = 64, 192, 6
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)
    try:
        if form == "int8":
            ctx.loadRouterInt8(0, *int8_router(0x3A, experts, d))
        else:
            ctx.loadRouter(0, synth.normal_bf16(0x3B, "warps.router", (experts, d), 0.02))
        x = hp.bf16_tensor(workload.make_tokens(0x3C, f"warps{rows}", rows, d), ctx.device)
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(2)]
        weights = [torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device) for _ in range(2)]
        logits = torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)
        router = hp.PrefillRouter(ctx)
        router.encodeGemma4Block(None, 0, x, got[0], weights[0], rows, outLogits=logits)
        router.encodeGemma4Block(None, 0, x, got[1], weights[1], rows)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        assert torch.equal(got[0], got[1])
        assert torch.equal(weights[0].view(torch.int16), weights[1].view(torch.int16))
    finally:
        ctx.close()


@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("experts,d,rows", [(9, 64, 17), (12, 4160, 24), (130, 3072, 25), (128, 6400, 160), (128, 6464, 160), (128, 2816, 161)])
def test_routes_of_a_short_chunk(form, experts, d, rows):
    """Edges of the one-launch kernel: tiles of eight rows and experts, contractions of more than one set of a warp's registers,
    and where the rows (160) or their width (fp32 rows of 6400) go over to the two launches.  Against blocks of 16 rows, twice
    in a row (its counters)."""
    from ane_fieldfare_b200 import hotpath as hp
    k = 5
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)
    try:
        eff = None if form == "bf16" else synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
        if form == "int8":
            ctx.loadRouterInt8(0, *int8_router(0x3D, experts, d), effectiveScale=eff)
        else:
            ctx.loadRouter(0, synth.normal_bf16(0x3E, "short.router", (experts, d), 0.02), effectiveScale=eff)
        x = hp.bf16_tensor(workload.make_tokens(0x3F, f"short{rows}", rows, d), ctx.device)
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(3)]
        weights = [torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device) for _ in range(3)]
        router = hp.PrefillRouter(ctx)
        for r in range(0, rows, 16):  # a block's kernel
            router.encodeGemma4Block(None, 0, x[r:], got[0][r:], weights[0][r:], min(16, rows - r))
        for i in (1, 2):
            router.encodeGemma4Block(None, 0, x, got[i], weights[i], rows)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        for i in (1, 2):
            assert torch.equal(got[0], got[i])
            assert torch.equal(weights[0].view(torch.int16), weights[i].view(torch.int16))
    finally:
        ctx.close()

@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("experts,d,rows", [(16, 6400, 160), (16, 6464, 160), (16, 12288, 40)])
def test_routes_of_a_short_chunk_of_few_experts(form, experts, d, rows):
    """The same at the widths' edge (fp32 rows of 6400) where the pairs of row and expert are few."""
    test_routes_of_a_short_chunk(form, experts, d, rows)


@pytest.mark.parametrize("form,experts,d,rows,one", [
    ("bf16", 128, 2816, 160, True), ("bf16", 256, 2816, 100, True), ("bf16", 256, 2816, 160, False), ("bf16", 256, 4096, 128, False),
    ("bf16", 128, 6144, 160, False), ("bf16", 256, 1024, 160, True), ("bf16_scaled", 128, 2816, 64, True),
    ("bf16_scaled", 128, 2816, 77, False), ("bf16_scaled", 128, 2816, 160, False), ("bf16_scaled", 128, 4096, 40, False),
    ("bf16_scaled", 128, 1024, 128, True), ("bf16_scaled", 16, 2816, 17, False), ("int8", 128, 2816, 77, True),
    ("int8", 128, 2816, 160, True), ("int8", 256, 2816, 160, False), ("int8", 128, 4096, 64, True), ("int8", 128, 4096, 128, False),
    ("int8", 128, 6144, 160, False)])
def test_short_chunks_take_the_shorter_way(form, experts, d, rows, one):
    """One launch or two, on 148 SMs, where the other was measurably slower (or no faster with weights from memory)."""
    from ane_fieldfare_b200 import hotpath as hp
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=8, maxTokens=rows)
    try:
        if ctx.info().smCount != 148:
            pytest.skip("measured on 148 SMs")
        eff = None if form == "bf16" else synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
        if form == "int8":
            ctx.loadRouterInt8(0, *int8_router(0x3D, experts, d), effectiveScale=eff)
        else:
            ctx.loadRouter(0, synth.normal_bf16(0x3E, "way.router", (experts, d), 0.02), effectiveScale=eff)
        x = hp.bf16_tensor(workload.make_tokens(0x3F, f"way{rows}", rows, d), ctx.device)
        ids = torch.zeros((rows, 8), dtype=torch.int32, device=ctx.device)
        weights = torch.zeros((rows, 8), dtype=torch.bfloat16, device=ctx.device)
        ctx.setTracing(True)
        hp.PrefillRouter(ctx).encodeGemma4Block(None, 0, x, ids, weights, rows)
        assert set(ctx.trace()) == ({"router_tile"} if one else {"router_approx", "router_select"})
    finally:
        ctx.close()


@pytest.mark.parametrize("form,experts,d,rows", [
    *[("bf16_scaled", 128, 4096, r) for r in (17, 33, 65, 97)], *[("int8", 256, 6464, r) for r in (17, 33, 65, 97)],
    *[("bf16", 256, 6464, r) for r in (33, 65, 97)]])
def test_selected_routes_of_small_token_tiles(form, experts, d, rows):
    """The two launches with token tiles of 32, 64, 96 and 128 rows."""
    from ane_fieldfare_b200 import hotpath as hp
    k = 8
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)
    try:
        load_router(ctx, form, experts, d)
        x = special_rows(hp, ctx, rows, d)
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(2)]
        weights = [torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device) for _ in range(2)]
        router = hp.PrefillRouter(ctx)
        for r in range(0, rows, 16):
            router.encodeGemma4Block(None, 0, x[r:], got[0][r:], weights[0][r:], min(16, rows - r), d + 8)
        ctx.setTracing(True)
        router.encodeGemma4Block(None, 0, x, got[1], weights[1], rows, d + 8)
        if ctx.info().smCount == 148:
            assert set(ctx.trace()) == {"router_approx", "router_select"}
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        assert torch.equal(got[0], got[1])
        assert torch.equal(weights[0].view(torch.int16), weights[1].view(torch.int16))
    finally:
        ctx.close()


@pytest.mark.parametrize("experts", [9, 131])
def test_logits_of_an_odd_number_of_experts(experts):
    """The kernel that forms every logit of many rows keeps each warp's rows aligned: ids as a block's kernel gives them."""
    from ane_fieldfare_b200 import hotpath as hp
    rows, d, k = 40, 192, 5
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)
    try:
        ctx.loadRouter(0, synth.normal_bf16(0x40, "odd.router", (experts, d), 0.02))
        x = hp.bf16_tensor(workload.make_tokens(0x41, "odd", rows, d), ctx.device)
        got = [torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device) for _ in range(2)]
        weights = torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device)
        logits = torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)
        router = hp.PrefillRouter(ctx)
        router.encodeGemma4Block(None, 0, x, got[0], weights, rows, outLogits=logits)
        for r in range(0, rows, 16):
            router.encodeGemma4Block(None, 0, x[r:], got[1][r:], weights[r:], min(16, rows - r))
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        assert torch.equal(got[0], got[1])
    finally:
        ctx.close()


@pytest.mark.parametrize("form", ["bf16", "bf16_scaled", "int8"])
@pytest.mark.parametrize("experts,d,rows", [(9, 64, 1), (16, 3072, 16), (16, 3136, 5), (128, 2816, 16), (256, 2880, 9), (256, 2880, 16),
                                            (160, 6208, 16), (130, 512, 13), (130, 576, 14)])
def test_block_router_at_its_edges(oracle, experts, d, rows, form):
    """A block's logits with one turn of a warp's chunks and more, one wave of CTAs and more: the oracle's, bit for bit."""
    from ane_fieldfare_b200 import hotpath as hp
    k = 5
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=16)
    try:
        x = workload.make_tokens(0x42, f"block{rows}", rows, d)
        eff = None if form == "bf16" else synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5))
        if form == "int8":
            router = int8_router(0x43, experts, d)
            ctx.loadRouterInt8(0, *router, effectiveScale=eff)
        else:
            router = synth.normal_bf16(0x41, "block.router", (experts, d), 0.02)
            ctx.loadRouter(0, router, effectiveScale=eff)
        ids = torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device)
        weights = torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device)
        logits = torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)
        hp.PrefillRouter(ctx).encodeGemma4Block(None, 0, hp.bf16_tensor(x, ctx.device), ids, weights, rows, outLogits=logits)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        if form == "int8":
            ref_ids, ref_w, ref_logits = oracle.router_topk_int8(*router, x, k, effective_scale=eff)
        else:
            ref_ids, ref_w, ref_logits = oracle.router_topk(
                oracle.LayerData(experts=np.zeros(16, dtype=np.uint8), stride=0, off=(0,) * 9, E=experts, D=d, F=64, K=k, router_w=router,
                                 router_scale=eff), x)
        assert np.array_equal(logits.cpu().numpy(), ref_logits)
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ref_ids)
        assert np.array_equal(hp.bf16_numpy(weights), ref_w)
    finally:
        ctx.close()


@pytest.mark.parametrize("d", [64, 512, 1088, 1536, 2304, 2816, 3584, 4672])
@pytest.mark.parametrize("experts,rows", [(10, 17), (256, 33)])
def test_int8_logits_of_many_rows(d, experts, rows):
    """Logits asked for, with one, two and three runs of a row held at a time and odd last runs: as blocks of 16 rows give them."""
    from ane_fieldfare_b200 import hotpath as hp
    k = 5
    ctx = hp.HotpathContext(layers=1, experts=experts, d=d, f=64, sharedF=0, topK=k, maxTokens=rows)
    try:
        ctx.loadRouterInt8(0, *int8_router(0x44, experts, d), effectiveScale=synth.bf16_bits(synth.uniform(7, d, 0.5, 1.5)))
        x = hp.bf16_tensor(workload.make_tokens(0x45, f"many{rows}", rows, d), ctx.device)
        got = [(torch.full((rows, k), -1, dtype=torch.int32, device=ctx.device), torch.zeros((rows, k), dtype=torch.bfloat16, device=ctx.device),
                torch.zeros((rows, experts), dtype=torch.float32, device=ctx.device)) for _ in range(2)]
        router = hp.PrefillRouter(ctx)
        for r in range(0, rows, 16):
            router.encodeGemma4Block(None, 0, x[r:], got[0][0][r:], got[0][1][r:], min(16, rows - r), outLogits=got[0][2][r:])
        router.encodeGemma4Block(None, 0, x, got[1][0], got[1][1], rows, outLogits=got[1][2])
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1].view(torch.int16), got[1][1].view(torch.int16))
        assert torch.equal(got[0][2], got[1][2])
    finally:
        ctx.close()
