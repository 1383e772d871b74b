"""Input rows with one value far above the rest whose weights are zero, at the sizes of the one-token kernel, the block
kernels and the GEMMs, against 64-bit sums: what is left of the row must keep its precision."""
import numpy as np
import pytest

from ane_fieldfare_b200 import gturbo, synth, workload
from test_gpu_router_int8 import int8_projection

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

D, F, COLUMN = 2816, 704, 5  # the outlier stands at an odd position, which has four bits fewer as digits


def f64(bits):
    return synth.bf16_to_float(bits).astype(np.float64)


def r16(v):
    return f64(synth.bf16_bits(v.astype(np.float32)))


def gelu(x):
    return 0.5 * x * (1.0 + np.tanh(np.clip(0.7978845608028654 * (x + 0.044715 * x ** 3), -20, 20)))


def error(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def rows_with_outlier(rows, power):
    x = f64(workload.make_tokens(0x92, f"outlier{rows}", rows, D)).reshape(rows, D)
    x[0::2, COLUMN] = 1.25 * 2.0 ** power
    return synth.bf16_bits(x.astype(np.float32)).reshape(rows, D)


def tolerance(zeros, power, scale, code):
    """The outputs' bf16 rounding, 2^-9 at most; where the weight is zero as code * scale + bias, the two parts, up to 24
    (INT4) or 255 scales large, are each rounded to 32 bits a few times before they cancel: an error `delta` relative to
    the rest of the row (2816 values, weights of about 0.03 for INT4 and 0.006 for INT8), in the gate and the up value.
    The activation's own rounding (steps of 2^-8 at most) turns it into whole steps: sqrt(delta 2^-8) in the mean square."""
    if zeros == "group":
        return 2.0 ** -9
    rest = np.sqrt(D) * (0.032 if code == 24 else 0.0055)
    delta = 4 * np.sqrt(2) * code * scale * 2.0 ** (power - 24) * 1.25 / rest
    return 2.0 ** -9 + delta + np.sqrt(delta * 2.0 ** -8)


def dequant4(blob, layout, name):
    w, s, b = gturbo.sub_tensor(blob, layout, name)
    rows, cols = layout.matrix_shape(name)
    w = w.reshape(rows, cols // 2)
    q = np.empty((rows, cols))
    q[:, 0::2], q[:, 1::2] = w & 15, w >> 4
    return q * np.repeat(f64(s).reshape(rows, -1), 64, 1) + np.repeat(f64(b).reshape(rows, -1), 64, 1)


@pytest.mark.parametrize("zeros,powers", [("group", (8, 12, 20, 30, 60)), ("column", (12, 16))])
def test_int4_rows(zeros, powers):
    from ane_fieldfare_b200 import hotpath as hp
    experts, k = 4, 2
    L = workload.make_layer(0x91, 0, experts=experts, d=D, f=F, sharedF=0, topK=k)
    L.blobs = L.blobs.copy()
    group = COLUMN // 64
    for e in range(experts):
        for name in ("gate", "up"):
            w, s, b = gturbo.sub_tensor(L.blobs[e], L.layout, name)
            w, s, b = w.reshape(F, D // 2), s.reshape(F, -1), b.reshape(F, -1)
            if zeros == "group":  # the whole group's
                s[:, group] = b[:, group] = 0
            else:  # the column's: code 8, bias -8 scales
                s[:, group], b[:, group] = synth.bf16_bits(np.float32([2.0 ** -7, -2.0 ** -4]))
                w[:, COLUMN // 2] = (w[:, COLUMN // 2] & 0x0F) | 0x80
    weights = [[dequant4(L.blobs[e], L.layout, n) for n in gturbo.ROLES] for e in range(k)]
    ctx = hp.HotpathContext(layers=1, experts=experts, d=D, f=F, sharedF=0, topK=k, maxTokens=16)
    try:
        workload.load_layer(ctx, 0, L)
        routed = hp.PrefillGroupedRoutedMoE(ctx)

        def partials(x, ids):
            p = torch.zeros((x.shape[0] * k, D), dtype=torch.bfloat16, device=ctx.device)
            routed.encodeVerifyBound(None, 0, hp.bf16_tensor(x, ctx.device), ids, p, x.shape[0])
            torch.cuda.synchronize()
            return hp.bf16_numpy(p).reshape(-1, k, D)

        for rows in (1, 2, 5, 16):
            ids = torch.tensor([[0, 1]] * rows, dtype=torch.int32, device=ctx.device)
            plain = synth.bf16_bits(f64(workload.make_tokens(0x92, f"outlier{rows}", rows, D)).astype(np.float32)).reshape(rows, D)
            without = partials(plain, ids)
            for power in powers:
                bits = rows_with_outlier(rows, power)
                x = f64(bits)
                want = np.stack([r16(gelu(x @ g.T) * (x @ u.T)) @ d.T for g, u, d in weights], axis=1)
                got = partials(bits, ids)
                tol = tolerance(zeros, power, 2.0 ** -7, 24)
                for t in range(0, rows, 2):
                    assert error(f64(got[t]), want[t]) < tol, (rows, power, t)
                assert np.array_equal(got[1::2], without[1::2])  # a row's bits do not depend on its neighbours
                if rows == 1:
                    one = torch.tensor([[1.0, 0.0]], dtype=torch.bfloat16, device=ctx.device)
                    y = torch.zeros((1, D), dtype=torch.bfloat16, device=ctx.device)
                    hp.MoE(ctx).encodeRoutedPersistentGPUSlots(None, 0, ids, hp.bf16_tensor(bits, ctx.device), one, None, y)
                    torch.cuda.synchronize()
                    assert error(f64(hp.bf16_numpy(y)), want[:, 0]) < tol, power
        assert ctx.info().deviceErrorFlag == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("zeros,powers", [("group", (12, 20, 30)), ("column", (12,))])
@pytest.mark.parametrize("rows", [1, 2, 5, 16, 40])
def test_int8_rows(zeros, powers, rows):
    from ane_fieldfare_b200 import hotpath as hp
    gate, up, down = (int8_projection(0x90, F, D, 0.5 / np.sqrt(D)), int8_projection(0x93, F, D, 0.5 / np.sqrt(D)),
                      int8_projection(0x96, D, F, 0.5 / np.sqrt(F)))
    for codes, s, b in (gate, up):
        if zeros == "group":
            s[:, 0] = b[:, 0] = 0
        else:
            s[:, 0], b[:, 0] = synth.bf16_bits(np.float32([2.0 ** -13, -2.0 ** -6]))
            codes[:, COLUMN] = 128
    g, u, d = (c * np.repeat(f64(s), 64, 1) + np.repeat(f64(b), 64, 1) for c, s, b in (gate, up, down))
    ctx = hp.HotpathContext(layers=1, experts=8, d=D, f=64, sharedF=F, topK=8, maxTokens=64)
    try:
        ctx.loadSharedInt8(0, gate, up, down)
        for power in powers:
            bits = rows_with_outlier(rows, power)
            x = f64(bits)
            want = r16(gelu(r16(x @ g.T)) * r16(x @ u.T)) @ d.T
            y = torch.zeros((rows, D), dtype=torch.bfloat16, device=ctx.device)
            hp.PrefillSharedExpert(ctx).encodeBlock(None, 0, hp.bf16_tensor(bits, ctx.device), y, rows)
            torch.cuda.synchronize()
            got = f64(hp.bf16_numpy(y))
            for t in range(0, rows, 2):
                assert error(got[t], want[t]) < tolerance(zeros, power, 2.0 ** -13, 255), (power, t)
        assert ctx.info().deviceErrorFlag == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("where", ["input", "activation"])
@pytest.mark.parametrize("rows", [1, 2, 7, 16])
def test_layer_with_shared_ffn(oracle, rows, where):
    """Routed experts and shared FFN of a layer call: the outlier's weights are zero everywhere, the oracle adds in fp32.
    activation: a feature whose up row is 2^20 times the others, its group's down weights zero."""
    from ane_fieldfare_b200 import hotpath as hp
    from conftest import assert_layer_close, oracle_layer
    d, f, fs, column = 1088, 192, 320, 70
    L = workload.make_layer(0x94, 0, experts=8, d=d, f=f, sharedF=fs, topK=3)
    L.blobs, L.sharedBlob = L.blobs.copy(), L.sharedBlob.copy()
    for blob, layout, width in [(b, L.layout, f) for b in L.blobs] + [(L.sharedBlob, L.sharedLayout, fs)]:
        for name in ("down",) if where == "activation" else ("gate", "up"):
            for part in gturbo.sub_tensor(blob, layout, name)[1:]:
                part.reshape(d if name == "down" else width, -1)[:, column // 64] = 0
        if where == "activation":
            for part in gturbo.sub_tensor(blob, layout, "up")[1:]:
                part.reshape(width, -1)[column] += np.uint16(20 << 7)
    x = workload.make_tokens(0x95, f"outlier.layer{rows}", rows, d).reshape(rows, d)
    if where == "input":
        L.routerW[:, column] = 0
        x[0::2, column] = synth.bf16_bits(np.float32([2.0 ** 24]))
    ctx = hp.HotpathContext(layers=1, experts=8, d=d, f=f, sharedF=fs, topK=3, maxTokens=16)
    try:
        workload.load_layer(ctx, 0, L)
        y = ctx.moeLayer(0, hp.bf16_tensor(x, ctx.device))
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want, *_ = oracle.moe_layer(oracle_layer(oracle, L), x, oracle.MODE_DECODE if rows == 1 else oracle.MODE_PARTIALS)
        rel_l2, _, _ = assert_layer_close(hp.bf16_numpy(y), want, oracle, f"outlier in the {where}, layer rows={rows}")
        assert rel_l2 < 2.0 ** -9  # both sides round the same sums to bf16: a share of neighbours, no more than the rounding itself
    finally:
        ctx.close()
