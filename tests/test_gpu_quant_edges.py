"""The quantisers where their fast paths hand over (f32 rows: two conversions per element, and comparisons for a group in which they
differ): elements within rounding distance of a mid-point, steps outside the range of the fast reciprocal; bf16 tensors, which are
compared throughout: elements at their thresholds, outputs too unaligned for the maximum's scratch words, one-row tensors.  Bit for
bit the oracle."""
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


@pytest.mark.parametrize('exp', [0, 20, -20])
@pytest.mark.parametrize('off', list(range(-12, 13, 2)) + [7, 9])
def test_bf16_elements_next_to_mid_points(off, exp):
    """Steps a few ulps off a short mantissa, so that mid-points times the step lie that close to bf16 numbers: there the
    thresholds rounded down to bf16 decide the packed comparisons."""
    P, O = pkg(), oracle()
    rng, N, K = np.random.default_rng(off + 100), 16, 512
    gs = np.array([(np.float32(2.0 ** -exp).view(np.int32) + off)], np.int32).view(np.float32)
    x = (rng.choice(np.concatenate([MID, [0, 0.5, 1, 6]]), (N, K // 16, 16)) * rng.choice([-1, 1], (N, K // 16, 16)) *
         rng.choice([1, 1.125, 1.5, 2, 3.25, 448], (N, K // 16, 1)) * 2.0 ** exp)
    x[:, :, 3] = 6 * np.abs(x).max(-1) / 6
    bits = O.f32_to_bf16_bits(x.astype(np.float32).reshape(N, K))
    bits = (bits.astype(np.int32) + rng.integers(-1, 2, bits.shape) * (rng.random(bits.shape) < 0.3)).clip(0, 0xffff).astype(bits.dtype)
    bits[(bits & 0x7f80) == 0x7f80] = 0
    W = P.quantize(to_dev_bf16(bits), gscale_in=torch.from_numpy(gs).cuda())
    p, s = O.quantize(O.bf16_bits_to_f32(bits), gs[0])
    assert np.array_equal(W.packed.cpu().numpy(), p) and np.array_equal(W.scale.cpu().numpy(), s)


@pytest.mark.parametrize('off', [0, 1])
def test_nan_weights_keep_their_zero_code(off):
    """A NaN exceeds no mid-point: code 0, its neighbours unaffected; aligned and unaligned rows, an odd number of groups."""
    P, O = pkg(), oracle()
    N, K = 3, 1040
    x = np.random.default_rng(8).normal(0, 0.02, (N, K)).astype(np.float32)
    bits = O.f32_to_bf16_bits(x)
    where = np.zeros((N, K), bool); where[0, 5] = where[1, 1030] = where[2, K - 1] = where[0, 0] = True
    clean = bits.copy(); clean[where] = 0
    bits[where] = 0x7fc0
    buf = torch.empty(N * K + 8, dtype=torch.bfloat16, device='cuda')
    w = buf[off:off + N * K].view(N, K)
    w.copy_(to_dev_bf16(bits))
    W = P.quantize(w)
    p, s, gs = O.quantize_tensor(O.bf16_bits_to_f32(clean))
    gp, gsc, ggs = W.numpy()
    assert np.array_equal(gp, p) and np.array_equal(gsc, s) and ggs.view(np.uint32)[0] == gs.view(np.uint32)[0]
