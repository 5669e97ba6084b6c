"""The quantisers where their fast paths hand over: elements within rounding distance of a mid-point, steps outside the range
of the fast reciprocal, outputs too unaligned for the maximum's scratch words, and one-row tensors.  Bit for bit the oracle."""
import numpy as np
import pytest
import torch

from util import pkg, oracle, to_dev_bf16

pytestmark = pytest.mark.gpu
MID = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], np.float32)


def check_rows(x):
    P, O = pkg(), oracle()
    p, s, gs = P.quantize_tokens(torch.from_numpy(x).cuda())
    rp, rs, rgs = O.quantize_rows(x)
    assert np.array_equal(gs.cpu().numpy().view(np.uint32), rgs.view(np.uint32))
    assert np.array_equal(s.cpu().numpy(), rs) and np.array_equal(p.cpu().numpy(), rp)


@pytest.mark.parametrize('scale', [1.0, 3e-5, 7.7e8, 1e-30, 1e33])
def test_elements_next_to_mid_points(scale):
    """Each group holds its maximum (6 steps exactly) and elements at a mid-point times the step, -3..3 ulps off, both signs."""
    K, rng = 1024, np.random.default_rng(3)
    x = np.empty((8, K), np.float32)
    for r in range(8):
        for g in range(K // 16):
            step = np.float32(scale * 2.0 ** (-(g % 7)) * (1 + g % 3 / 8))
            v = np.nextafter((MID[rng.integers(0, 7, 16)] * step).astype(np.float32), np.float32(0))
            for _ in range(rng.integers(0, 4)):
                v = np.nextafter(v, np.float32(np.inf)).astype(np.float32)
            x[r, 16 * g:16 * g + 16] = v * np.where(rng.random(16) < 0.5, -1, 1)
            x[r, 16 * g + g % 16] = 6 * step
    check_rows(x)


def test_more_rows_than_the_cta_per_row_kernel_takes():
    """Wide GEMM products of many f32 rows (a warp quantises a row) equal those of the same rows a few at a time."""
    P = pkg()
    g = torch.Generator(device='cuda').manual_seed(5)
    for K in (256, 768, 1536, 2048):
        W = P.quantize((torch.randn((64, K), generator=g, device='cuda') * 0.02).to(torch.bfloat16))
        x = torch.randn((2500, K), generator=g, device='cuda') * torch.exp(torch.randn((2500, 1), generator=g, device='cuda'))
        x[7] = 0; x[9, 3] = float('inf')
        y = P.gemm(W, x, ws=P.split_workspace(2500, K, 'cuda'))
        for m0 in (0, 1000, 2484):
            sub = x[m0:m0 + 16].contiguous()
            ys = P.gemm(W, sub, ws=P.split_workspace(16, K, 'cuda'))
            assert torch.equal(ys.view(torch.int32), y[m0:m0 + 16].contiguous().view(torch.int32)), (K, m0)


@pytest.mark.parametrize('N,K,off', [(1, 16, 0), (3, 48, 1), (300, 272, 2), (513, 1040, 0)])
def test_quantize_with_unaligned_outputs(N, K, off):
    P, O = pkg(), oracle()
    bits = O.f32_to_bf16_bits(np.random.default_rng(N).normal(0, 0.02, (N, K)).astype(np.float32))
    buf = torch.full((N * K // 2 + 8,), 255, dtype=torch.uint8, device='cuda')
    out = P.Nvfp4Weight(torch.zeros((N, K // 2)), torch.zeros((N, K // 16)), torch.full((1,), 7.0))
    out.packed = buf[off:off + N * K // 2].view(N, K // 2)
    W = P.quantize(to_dev_bf16(bits), out=out)
    p, s, gs = O.quantize_tensor(O.bf16_bits_to_f32(bits))
    gp, gsc, ggs = W.numpy()
    assert np.array_equal(gp, p) and np.array_equal(gsc, s) and ggs.view(np.uint32)[0] == gs.view(np.uint32)[0]
