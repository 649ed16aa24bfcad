"""Kernel forms chosen by a step's sizes, at the sizes where one takes over from another, against the references of the general forms."""
import pytest
import torch

from blaze_b200 import quant
from blaze_b200.batch import SeqChunk, build_batch
from blaze_b200.config import ModelConfig, RopeConfig, inv_freq
from blaze_b200.kv import KVCache
from blaze_b200.linear import Linear
from blaze_b200.ops import ref
from blaze_b200.quant import Format
from test_gpu_kernels import _A, _attention_case, _experts, ops       # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("M", [1, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(128, 128), (200, 384), (1024, 5120), (5120, 8192), (40000, 256)])
def test_fp8_block_product_of_few_rows(ops, M, N, K):      # noqa: F811
    """Rows on the MMA's columns and K over a cluster, against the stored codes and scales in 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(11)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    lin = Linear.from_dense(torch.randn(N, K, generator=g, device=DEV) * 0.02, Format.FP8_BLOCK)
    lin.bias = torch.randn(N, generator=g, device=DEV).bfloat16()
    q, sc = ops.quantize_fp8_block(x)
    got = ops.linear(lin, x, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert ops.take_status() == 0
    xd = (q.view(torch.float8_e4m3fn).double().view(M, K // 128, 128) * sc[:, :M].t().double().unsqueeze(-1)).view(M, K)
    assert _rel(got, xd @ lin.dequant().double().t() + lin.bias.double()) < 1e-5
    assert torch.equal(ops.linear(lin, x), got.bfloat16())      # and the same sums when they are rounded
