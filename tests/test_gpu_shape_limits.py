"""Model shapes at the limits of the small-row kernels' shared memory, against the CPU oracle: one row through the
layer call, its host form, the stack and the separate operators, for shapes that fill the one-token kernel and for
shapes past it (which take the block kernels)."""
import numpy as np
import pytest

from ane_fieldfare_b200 import workload
from conftest import LAYER_ELEMENTWISE_TOL, assert_layer_close, oracle_layer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def context(L, rows):
    from ane_fieldfare_b200 import hotpath as hp
    ctx = hp.HotpathContext(layers=1, experts=L.experts, d=L.d, f=L.f, sharedF=L.sharedF, topK=L.topK, maxTokens=rows)
    workload.load_layer(ctx, 0, L)
    return hp, ctx


@pytest.mark.parametrize("d,f,fs,k,launches", [
    (2816, 704, 2816, 8, 1), (2880, 704, 2112, 8, 1), (3072, 704, 2112, 8, 1), (2816, 896, 0, 8, 1),
    (2560, 1024, 0, 8, 1), (3968, 64, 0, 7, 1),
    # past one CTA's shared memory: router, gate/up, down, combine
    (2880, 1024, 2112, 8, 4), (1856, 1024, 4800, 8, 4), (3904, 192, 960, 3, 4), (4096, 512, 0, 8, 4)])
def test_one_row(oracle, d, f, fs, k, launches):
    L = workload.make_layer(0x81, 0, experts=16, d=d, f=f, sharedF=fs, topK=k)
    hp, ctx = context(L, 1)
    try:
        ld = oracle_layer(oracle, L)
        x = workload.make_tokens(0x82, "limits", 1, d)
        xd = hp.bf16_tensor(x, ctx.device)
        want, _, ref_ids, ref_w = oracle.moe_layer(ld, x, oracle.MODE_DECODE)
        ids = torch.full((1, k), -1, dtype=torch.int32, device=ctx.device)
        before = ctx.info().kernelLaunches
        y = ctx.moeLayer(0, xd, ids=ids)
        torch.cuda.synchronize()
        assert ctx.info().kernelLaunches - before == launches
        assert np.array_equal(ids.cpu().numpy().astype(np.uint32), ref_ids)
        assert_layer_close(hp.bf16_numpy(y), want, oracle, f"one row {d}x{f}+{fs}", elementwise_tol=LAYER_ELEMENTWISE_TOL)
        host = torch.empty((1, d), dtype=torch.bfloat16).pin_memory()
        ctx.moeLayerHost(0, xd.cpu().pin_memory(), host)
        assert torch.equal(host, y.cpu())
        # the operators one by one: the same bits; the shared FFN is the routed part's residual
        shared = None
        if fs:
            shared = torch.zeros((1, d), dtype=torch.bfloat16, device=ctx.device)
            hp.SharedExpertInt4(ctx).encode(None, 0, xd, shared)
        weights = hp.bf16_tensor(ref_w.reshape(1, k), ctx.device)
        parts = torch.zeros_like(y)
        moe = hp.MoE(ctx)
        moe.encodeRouterGemma4(None, 0, xd, ids, weights, topK=k)
        moe.encodeRoutedPersistentGPUSlots(None, 0, ids, xd, weights, shared, parts)
        assert torch.equal(parts, y)
        # given routes may repeat an expert; one past the experts is dropped and reported
        ids[0, 1:] = ids[0, 0]
        moe.encodeRoutedPersistentGPUSlots(None, 0, ids, xd, weights, None, parts)
        e = int(ref_ids[0, 0])
        v = oracle.expert_ffn(L.blobs[e], L.layout.offsets.as_tuple(), d, f, x)[0].astype(np.float64)
        total = oracle.bf16_to_float(hp.bf16_numpy(weights)).astype(np.float64).sum() * v
        got = oracle.bf16_to_float(hp.bf16_numpy(parts))[0]
        assert np.linalg.norm(got - total) <= 1e-2 * np.linalg.norm(total)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        one = ids.clone()
        one[0, 1:] = 16
        moe.encodeRoutedPersistentGPUSlots(None, 0, one, xd, weights, None, parts)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 12
        ctx.resetDeviceError()
        only = oracle.bf16_to_float(hp.bf16_numpy(weights))[0, 0].astype(np.float64) * v
        got = oracle.bf16_to_float(hp.bf16_numpy(parts))[0]
        assert np.linalg.norm(got - only) <= 1e-2 * np.linalg.norm(only)
    finally:
        ctx.close()


@pytest.mark.parametrize("d,f,fs,k", [(64, 11072, 0, 2), (64, 64, 21376, 2), (128, 16384, 11136, 3)])
@pytest.mark.parametrize("rows", [2, 3, 5, 16])
def test_wide_blocks(oracle, d, f, fs, k, rows):
    """Widths whose rows fit as digits two at a time, not four."""
    L = workload.make_layer(0x83, 0, experts=6, d=d, f=f, sharedF=fs, topK=k)
    hp, ctx = context(L, 16)
    try:
        x = workload.make_tokens(0x84, f"wide{rows}", rows, d)
        y = ctx.moeLayer(0, hp.bf16_tensor(x, ctx.device))
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want, *_ = oracle.moe_layer(oracle_layer(oracle, L), x, oracle.MODE_PARTIALS)
        assert_layer_close(hp.bf16_numpy(y), want, oracle, f"wide block {d}x{f}+{fs} rows={rows}")
    finally:
        ctx.close()
