"""NVFP4 quantisers and the block-scaled tcgen05 GEMM against the PyTorch emulation of the format."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ext():
    from surogate_b200.ops import ext as load

    return load()


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("rows,K,block2d", [(128, 256, False), (200, 512, False), (256, 256, True), (384, 1024, True)])
def test_quantize_rows_matches_emulation(ext, rows, K, block2d):
    from surogate_b200.ops import nvfp4_ref as ref

    torch.manual_seed(0)
    x = (torch.randn(rows, K, device=DEV) * torch.rand(rows, 1, device=DEV) * 3).bfloat16()
    amax = x.float().abs().max().reshape(1)
    q, sf = ext.nvfp4_quantize(x, amax, False, 0, block2d)
    codes, sfd, ge = ref.quantize(x.float(), amax[0], block2d)
    sf_k = ref.atoms_to_sf(sf, rows, K // 16)
    sf_got = sf_k.view(torch.float8_e4m3fn).float()
    # a scale that sits on an e4m3 rounding boundary may round the other way (different operation order): rare, one ulp
    sf_bad = (sf_got != sfd)
    assert sf_bad.float().mean().item() < 5e-3
    assert ((sf_got - sfd).abs() <= 0.13 * sfd + 1e-6).all()
    got = ref.unpack_codes(q)
    ok_blocks = (~sf_bad).repeat_interleave(16, dim=1)
    mismatch = ((got != codes) & ok_blocks).float().mean().item()
    assert mismatch < 2e-3, mismatch   # products can land on a rounding boundary differently
    deq = ext.nvfp4_dequantize(q, sf, amax, 1.0)
    assert _rel(deq, ref.dequantize(got, sf_got, ge)) < 4e-3
    assert _rel(deq, x) < 0.15


def test_quantize_transpose_and_hadamard(ext):
    from surogate_b200.ops import nvfp4_ref as ref

    torch.manual_seed(1)
    R, C = 256, 192
    x = torch.randn(R, C, device=DEV).bfloat16()
    amax = x.float().abs().max().reshape(1)
    q, sf = ext.nvfp4_quantize_transpose(x, amax, False, False, 0, 0)
    codes, sfd, ge = ref.quantize(x.float().t().contiguous(), amax[0])
    sf_got = ref.atoms_to_sf(sf, C, R // 16).view(torch.float8_e4m3fn).float()
    sf_bad = sf_got != sfd
    assert sf_bad.float().mean().item() < 5e-3
    assert (((ref.unpack_codes(q) != codes) & (~sf_bad).repeat_interleave(16, dim=1)).float().mean().item()) < 2e-3
    # random Hadamard: quantised transform de-quantises back to (approximately) the transform of x^T
    mask = 0b1011001110001101
    q2, sf2 = ext.nvfp4_quantize_transpose(x, amax, False, True, 0, mask)
    deq = ext.nvfp4_dequantize(q2, sf2, amax, 2.0)
    want = ref.hadamard16(x.float().t().contiguous(), mask)
    assert _rel(deq, want) < 0.13
    # the transform is orthonormal: products along the transformed dimension are preserved
    y = torch.randn(R, 64, device=DEV).bfloat16()
    hy = ref.hadamard16(y.float().t().contiguous(), mask)
    assert _rel(want @ hy.t(), x.float().t() @ y.float()) < 1e-3


def test_stochastic_rounding_is_unbiased(ext):
    x = torch.full((128, 256), 0.7, device=DEV).bfloat16()
    x[:, ::16] = 6.0   # pins every block scale so that 0.7 falls strictly between two grid points
    amax = torch.tensor([6.0], device=DEV)
    acc = torch.zeros(128, 256, device=DEV)
    n = 32
    for seed in range(n):
        q, sf = ext.nvfp4_quantize(x, amax, True, seed, False)
        acc += ext.nvfp4_dequantize(q, sf, amax, 1.0).float()
    mean = (acc / n)[:, 1:16].mean().item()
    assert abs(mean - 0.7) < 0.02, mean
    q, sf = ext.nvfp4_quantize(x, amax, False, 0, False)
    rn = ext.nvfp4_dequantize(q, sf, amax, 1.0).float()[:, 1:16].mean().item()
    assert abs(rn - 0.7) > 0.04   # round-to-nearest is biased on this input


@pytest.mark.parametrize("M,N,K", [(128, 128, 256), (256, 384, 512), (1024, 768, 2048), (300, 264, 768)])
def test_gemm_nvfp4(ext, M, N, K):
    torch.manual_seed(2)
    a = (torch.randn(M, K, device=DEV) * (1 + torch.rand(M, 1, device=DEV))).bfloat16()
    b = (torch.randn(N, K, device=DEV) * (1 + torch.rand(N, 1, device=DEV))).bfloat16()
    am_a, am_b = a.float().abs().max().reshape(1), b.float().abs().max().reshape(1)
    qa, sfa = ext.nvfp4_quantize(a, am_a, False, 0, False)
    qb, sfb = ext.nvfp4_quantize(b, am_b, False, 0, False)
    da, db = ext.nvfp4_dequantize(qa, sfa, am_a, 1.0), ext.nvfp4_dequantize(qb, sfb, am_b, 1.0)
    ref = da.float() @ db.float().t()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    inv_a, inv_b = am_a / 2688.0, am_b / 2688.0
    ext.gemm_nvfp4(qa, sfa, qb, sfb, out, False, 1.0, inv_a, inv_b, ext.error_flag_tensor())
    torch.cuda.synchronize()
    assert ext.read_error_flag(True) == 0
    assert _rel(out, ref) < 8e-3, _rel(out, ref)
    assert _rel(out, a.float() @ b.float().t()) < 0.2


@pytest.mark.parametrize("rows,K,block2d", [(256, 512, False), (512, 1024, True)])
def test_four_over_six_matches_the_codec_emulation_and_lowers_the_error(ext, rows, K, block2d):
    """The four-over-six quantiser (per block: abs-max -> 6 or abs-max -> 4, whichever reconstructs better; tensor encode factor
    1536) against the PyTorch emulation in quant/codecs.py for 1-D blocks, and against the plain quantiser's error for both kinds."""
    from surogate_b200.quant.codecs import NVFP4Storage

    torch.manual_seed(1)
    x = (torch.randn(rows, K, device=DEV) * torch.rand(rows, 1, device=DEV) * 3).bfloat16()
    amax = x.float().abs().max().reshape(1)
    q, sf = ext.nvfp4_quantize(x, amax, False, 0, block2d, True)
    deq = ext.nvfp4_dequantize(q, sf, amax, 1.0, 1536.0)
    q0, sf0 = ext.nvfp4_quantize(x, amax, False, 0, block2d, False)
    deq0 = ext.nvfp4_dequantize(q0, sf0, amax, 1.0)
    e46, e6 = _rel(deq, x), _rel(deq0, x)
    # a few per cent lower on Gaussian data with 1-D blocks; a 16 x 16 tile shares one scale among 256 values, where the choice rarely matters
    assert e46 < e6 * (1.001 if block2d else 0.97), (e46, e6)
    from surogate_b200.ops import nvfp4_ref as ref

    sf_val = ref.atoms_to_sf(sf, rows, K // 16).view(torch.float8_e4m3fn).float()                      # decoded block scales [rows, K/16]
    blk_amax = x.float().abs().reshape(rows, K // 16, 16).amax(-1)
    if block2d:
        blk_amax = blk_amax.reshape(rows // 16, 16, K // 16).amax(1, keepdim=True).expand(rows // 16, 16, K // 16).reshape(rows, K // 16)
    sf_if_6 = blk_amax * (1536.0 / amax) / 6.0
    picked4 = (sf_val > 1.25 * sf_if_6).float().mean().item()                                            # the other mapping gives 1.5 x that scale
    assert (0.0 if block2d else 0.02) <= picked4 < 0.98, picked4       # both mappings are in use
    if not block2d:
        codec = NVFP4Storage(four_over_six=True)
        st = codec.quantize(x.reshape(-1))
        emu = codec.dequantize_reference(st).reshape(rows, K)
        assert _rel(deq, emu) < 2e-2, _rel(deq, emu)   # same algorithm; ties and e4m3 rounding order may differ on a few blocks
    # stochastic rounding ignores the flag (gradients keep the plain mapping and the 2688 factor)
    qs, sfs = ext.nvfp4_quantize(x, amax, True, 5, False, True)
    assert _rel(ext.nvfp4_dequantize(qs, sfs, amax, 1.0), x) < 0.25


def test_gemm_with_four_over_six_operands(ext):
    torch.manual_seed(2)
    M, N, K = 256, 384, 512
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = torch.randn(N, K, device=DEV).bfloat16()
    am_a, am_b = a.float().abs().max().reshape(1), b.float().abs().max().reshape(1)
    qa, sfa = ext.nvfp4_quantize(a, am_a, False, 0, False, True)
    qb, sfb = ext.nvfp4_quantize(b, am_b, False, 0, True, True)
    d = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ext.gemm_nvfp4(qa, sfa, qb, sfb, d, False, 1.0, am_a / 1536.0, am_b / 1536.0, ext.error_flag_tensor())
    da, db = ext.nvfp4_dequantize(qa, sfa, am_a, 1.0, 1536.0), ext.nvfp4_dequantize(qb, sfb, am_b, 1.0, 1536.0)
    assert _rel(d, da.float() @ db.float().t()) < 6e-3
    assert _rel(d, a.float() @ b.float().t()) < 0.2


def _sr_codes(s, seed, idx):
    """Stochastic rounding as the kernels define it: splitmix64 of the element index gives u in [0, 1); the upper grid neighbour is
    taken when u is below the position between the neighbours."""
    import numpy as np

    z = idx.astype(np.uint64) + np.uint64((0x9E3779B97F4A7C15 * (seed + 1)) % 2 ** 64)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    u = (z >> np.uint64(40)).astype(np.float64) / 2.0 ** 24
    grid = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
    a = np.minimum(np.abs(s.astype(np.float64)), 6.0)
    lo = np.searchsorted(grid, a, side="right") - 1
    nxt = np.minimum(lo + 1, 7)
    p = (a - grid[lo]) / np.maximum(grid[nxt] - grid[lo], 0.5)
    return np.where(u < p, nxt, lo) + 8 * (s < 0)


@pytest.mark.parametrize("transpose,rows,K", [(False, 16, 16), (False, 129, 48), (False, 200, 400), (False, 384, 272),
                                              (True, 64, 64), (True, 192, 320), (True, 320, 192)])
@pytest.mark.parametrize("stochastic", [False, True])
def test_quantisers_at_the_edges_of_their_tiles(ext, transpose, rows, K, stochastic):
    """Sizes below, between and just above the 128 x 128 tiles (`rows` x `K` is the quantised shape): codes against the emulation, and
    zero scales in the padding rows and blocks, which the tensor core reads."""
    import numpy as np
    from surogate_b200.ops import nvfp4_ref as ref

    torch.manual_seed(rows + K)
    x = (torch.randn(rows, K, device=DEV) * torch.rand(rows, 1, device=DEV) * 3).bfloat16()
    x[0, 0] = -0.0
    amax = x.float().abs().max().reshape(1)
    q, sf = ext.nvfp4_quantize_transpose(x.t().contiguous(), amax, stochastic, False, 11, 0) if transpose else ext.nvfp4_quantize(x, amax, stochastic, 11, False)
    codes, sfd, ge = ref.quantize(x.float(), amax[0])
    sf_all = ref.atoms_to_sf(sf, (rows + 127) // 128 * 128, (K // 16 + 3) // 4 * 4)
    sf_got = sf_all[:rows, :K // 16].view(torch.float8_e4m3fn).float()
    assert not sf_all[rows:].any() and not sf_all[:, K // 16:].any()
    sf_bad = sf_got != sfd
    assert sf_bad.float().mean().item() < 5e-3
    if stochastic:
        s = (x.float().view(rows, -1, 16) * torch.where(sfd > 0, ge / sfd, torch.zeros_like(sfd)).unsqueeze(-1)).view(rows, K).cpu().numpy()
        idx = np.arange(rows * K, dtype=np.uint64).reshape(rows, K)
        codes = torch.from_numpy(_sr_codes(s, 11, idx).astype(np.int64)).to(DEV)
    wrong = (ref.unpack_codes(q) != codes) & (~sf_bad).repeat_interleave(16, dim=1)
    assert wrong.float().mean().item() < 2e-3       # a product on a rounding boundary may fall the other way


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("hadamard", [False, True])
def test_stochastic_codes_do_not_depend_on_the_tile_height(ext, transpose, hadamard):
    """Tensors of at most one 128 x 128 tile per SM are quantised in tiles of 32 rows, larger ones in whole tiles (19 x 8 of them here): the same
    codes and scales, since the random numbers belong to the element."""
    if hadamard and not transpose:
        pytest.skip("the Hadamard transform is part of the transposing quantiser")
    torch.manual_seed(7)
    rows, K, part = 2432, 1024, 1280
    x = (torch.randn(rows, K, device=DEV) * 2).bfloat16()
    amax = x.float().abs().max().reshape(1)

    def quantise(t):
        if transpose:
            return ext.nvfp4_quantize_transpose(t.t().contiguous(), amax, True, hadamard, 5, 0xB2CD)
        return ext.nvfp4_quantize(t.contiguous(), amax, True, 5, False)

    q, sf = quantise(x)
    qp, sfp = quantise(x[:part])
    assert torch.equal(q[:part], qp) and torch.equal(sf[:sfp.numel()], sfp) and part % 128 == 0
    if not transpose:
        assert torch.equal(ext.nvfp4_quantize(x, amax, True, 5, True)[0][:part], ext.nvfp4_quantize(x[:part], amax, True, 5, True)[0])
