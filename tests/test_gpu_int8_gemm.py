"""The INT8 shared FFN's tensor-core GEMM (more than 16 rows) against the oracle at the edges of its
token tiles (32, 64, 96, 128 columns), with a row stride, and at widths whose tiles pair unevenly."""
import numpy as np
import pytest

from ane_fieldfare_b200 import workload
from conftest import ELEMENTWISE_TOL, assert_layer_close
from test_gpu_router_int8 import int8_projection

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d,fs", [(128, 192), (448, 64), (4160, 320), (2816, 2112)])
@pytest.mark.parametrize("rows", [17, 32, 33, 96, 128, 129, 300])
def test_int8_gemm_edges(oracle, d, fs, rows):
    from ane_fieldfare_b200 import hotpath as hp
    gate, up = int8_projection(0x90, fs, d, 0.5 / np.sqrt(d)), int8_projection(0x93, fs, d, 0.5 / np.sqrt(d))
    down = int8_projection(0x96, d, fs, 0.5 / np.sqrt(fs))
    ctx = hp.HotpathContext(layers=1, experts=8, d=d, f=64, sharedF=fs, topK=8, maxTokens=300)
    try:
        ctx.loadSharedInt8(0, gate, up, down)
        x = workload.make_tokens(0x2B, f"int8.gemm{rows}", rows, d)
        wide = torch.zeros((rows, d + 8), dtype=torch.bfloat16, device=ctx.device)
        wide[:, :d] = hp.bf16_tensor(x, ctx.device)
        y = torch.zeros((rows, d), dtype=torch.bfloat16, device=ctx.device)
        hp.PrefillSharedExpert(ctx).encodeBlock(None, 0, wide, y, rows, hiddenStrideElements=d + 8)
        torch.cuda.synchronize()
        assert ctx.info().deviceErrorFlag == 0
        want = oracle.shared_ffn_int8(gate, up, down, x)
        assert_layer_close(hp.bf16_numpy(y), want, oracle, f"int8 gemm {d}x{fs} rows={rows}",
                           elementwise_tol=ELEMENTWISE_TOL)
        assert np.mean(hp.bf16_numpy(y) != want) < 2e-2
    finally:
        ctx.close()
