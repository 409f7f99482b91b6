"""The register-resident quantisers: codes against the division they replace, every width class, odd rows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _codes(x):
    """clamp(rne(x / s)) and s as the oracle states them (fp32 division), on the GPU; NaN -> -128."""
    amax = torch.nan_to_num(x.float().abs(), nan=0.0, posinf=math.inf).amax(1)
    s = torch.where(amax > 0, amax / torch.full_like(amax, 127.0), torch.ones_like(amax))
    q = torch.round(x.float() / s[:, None]).clamp(-128, 127)
    return torch.where(torch.isnan(q), torch.full_like(q, -128.0), q).to(torch.int8), s


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 248), (2, 512), (5, 1024), (16, 4096), (64, 5120), (7, 8200), (2, 11008), (1, 16384),
                                       (600, 512), (513, 4096), (700, 1000)])
def test_codes_of_plain_rows(rows, cols):
    from lsvd_b200.ffn import act_quant
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, generator=g, device="cuda") * torch.logspace(-7, 4, rows, device="cuda")[:, None]
    x = x.clamp(-60000, 60000).half()
    if rows > 2:
        x[1] = 0
        x[2, 0], x[2, 1], x[2, -1] = math.inf, -math.inf, math.nan
        x[0, 0] = math.nan
    q, s, _ = act_quant(x)
    q_ref, s_ref = _codes(x)
    assert torch.equal(s, s_ref)
    assert torch.equal(q, q_ref)


def test_codes_equal_the_division_on_every_magnitude():
    """Each fp16 magnitude against scales of many rows: 31 000 values x 512 scales, no code differs from the division."""
    from lsvd_b200.ffn import act_quant
    vals = torch.arange(1, 0x7bff, 2, dtype=torch.int16, device="cuda").view(torch.float16)      # positive finite values
    rows = 512
    g = torch.Generator(device="cuda").manual_seed(5)
    x = vals[torch.randint(0, vals.numel(), (rows, 16384), generator=g, device="cuda")]
    top = torch.logspace(-6, 4.8, rows, device="cuda").half()
    x = torch.minimum(x, top[:, None]) * torch.where(torch.rand(x.shape, generator=g, device="cuda") < 0.5, -1, 1).half()
    x[:, 0] = top
    q, s, _ = act_quant(x)
    q_ref, s_ref = _codes(x)
    assert torch.equal(s, s_ref) and torch.equal(q, q_ref)


@pytest.mark.parametrize("rows,cols", [(1, 64), (16, 4096), (3, 5120), (2, 12000), (520, 4096)])
def test_rmsnorm_rows(rows, cols):
    """fp32 statistics in any order: an fp32 mean is off by a few ulp, far below an fp16 step, so x * inv rounds to the 64-bit
    fp16 number or its neighbour.  One step of that number, times the weight, is at most two steps of the product (the steps
    of neighbouring binades differ by two), and rounding both products moves them by half a step each: three steps.  Few
    entries move at all; the codes follow from the row exactly."""
    from lsvd_b200.ffn import act_quant
    g = torch.Generator(device="cuda").manual_seed(cols)
    x, w = torch.randn(rows, cols, generator=g, device="cuda").half(), (1 + 0.1 * torch.randn(cols, generator=g, device="cuda")).half()
    q, s, xn = act_quant(x, want_rotated=True, norm_weight=w, norm_eps=1e-5)
    inv = torch.rsqrt(x.double().square().mean(1, keepdim=True) + 1e-5)
    ref = ((x.double() * inv).half().double() * w.double()).half()
    step = 2.0 ** (torch.floor(torch.log2(ref.double().abs().clamp_min(2 ** -14))) - 10)
    assert bool(((xn.double() - ref.double()).abs() <= 3 * step).all())
    assert float((xn != ref).float().mean()) < 1e-2
    q_ref, s_ref = _codes(xn)
    assert torch.equal(s, s_ref) and torch.equal(q, q_ref)


@pytest.mark.parametrize("rows,cols", [(300, 8), (300, 264), (200, 1000), (100, 4096), (60, 5120), (40, 8200), (40, 16384)])
def test_rmsnorm_of_a_row_does_not_depend_on_its_alignment(rows, cols):
    """A row at a 2-byte boundary takes the routine that the fused kernel also runs, an aligned one the register-resident
    kernel: the squares are added in one order, so the statistics, rows, scales and codes are the same bits."""
    from lsvd_b200.ffn import act_quant
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x, w = torch.randn(rows, cols, generator=g, device="cuda").half(), (1 + 0.1 * torch.randn(cols, generator=g, device="cuda")).half()
    odd = torch.empty(rows, cols + 1, dtype=torch.float16, device="cuda")[:, 1:]
    odd.copy_(x)
    for a, b in zip(act_quant(x, want_rotated=True, norm_weight=w, norm_eps=1e-5), act_quant(odd, want_rotated=True, norm_weight=w, norm_eps=1e-5)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("rows", [1, 5, 149, 700, 2500])
@pytest.mark.parametrize("K,nb", [(12, 64), (16, 64), (28, 64), (32, 64), (60, 64), (108, 64), (172, 64), (12, 128), (28, 128), (60, 128), (108, 128),
                                  (172, 128)])
def test_one_token_per_block_rotation(rows, K, nb):
    """Against the oracle's rotation on the CPU: had_K is +-1 and the sums of up to 172 fp16 values are taken in fp32 in another
    order, so a result may round the other way (one fp16 step); codes and scale follow from the rotated row exactly.  The
    batch form and the throughput form (more rows than SMs) give the same bits."""
    from lsvd_b200.ffn import hadamard_pack, hadamard_quant
    from oracle import ffn as offn
    g = torch.Generator().manual_seed(K + nb + rows)
    hk = (torch.randint(0, 2, (K, K), generator=g) * 2 - 1).float()
    x = torch.randn(rows, K * nb, generator=g).half()
    packed = hadamard_pack(hk.half().cuda())
    q, s, y = hadamard_quant(x.cuda(), packed, K, want_rotated=True)
    ref = offn.hadamard_full(x[:8], hk, K)
    step = 2.0 ** (torch.floor(torch.log2(ref.double().abs().clamp_min(2 ** -14))) - 10)
    assert bool(((y[:8].cpu().double() - ref.double()).abs() <= step).all())
    q_ref, s_ref = _codes(y)
    assert torch.equal(s, s_ref) and torch.equal(q, q_ref)
    few = hadamard_quant(x[-3:].contiguous().cuda(), packed, K)
    assert torch.equal(few[0], q[-3:]) and torch.equal(few[1], s[-3:])
    odd = torch.zeros(rows, K * nb + 2, dtype=torch.int8, device="cuda")[:, 2:]               # rows at 2-byte alignment
    hadamard_quant(x.cuda(), packed, K, q=odd)
    assert torch.equal(odd, q)
