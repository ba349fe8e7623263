"""Gates of a Gated DeltaNet prompt portion in one kernel (csrc/kernels/gdn_ab_gates.cu), and the convolution beside it at the edges of
its runs of tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens around the 16 of a cluster; inputs from one chunk of 32 (31 of 32 warps idle) to the benchmark's 5120; heads with and without
# all eight feature groups
@pytest.mark.parametrize("t,h,hv", [(1, 32, 4), (15, 160, 32), (16, 1024, 6), (17, 5120, 32), (40, 5120, 32), (333, 2080, 16), (2047, 256, 3)])
def test_gates_match_the_projection_and_the_gates_apart(t, h, hv):
    from deepseek_v4_2080ti_b200.ops import basic, gdn
    torch.manual_seed(t)
    x = torch.randn(t, h, device="cuda").bfloat16()
    w = (torch.randn(2 * hv, h, device="cuda") * h ** -0.5).bfloat16()
    a_log, dt = torch.randn(hv, device="cuda") * 0.5, torch.randn(hv, device="cuda")
    assert gdn.ab_gates_fit(t, h, hv)
    g, beta = gdn.ab_gates(x, w, a_log, dt, hv)
    exact = x.double() @ w.double().t()
    ab = exact.bfloat16()
    g_ref, b_ref = basic.gdn_gates(ab, 0, hv, a_log, dt, hv)
    # fp32 sums in another order than 64 bits may round to the neighbouring bf16 value (2^-7 of it at most, and 2^-20 where the sum
    # cancels); softplus has slope 1 at most, the sigmoid 1/4; fast exponentials and logarithms agree to 1e-5
    step = exact.abs() * 2.0 ** -7 + 2.0 ** -20
    assert ((g - g_ref).abs() <= a_log.exp() * step[:, :hv] + 1e-5 * g_ref.abs()).all()
    assert ((beta - b_ref).abs() <= step[:, hv:] / 4 + 1e-5).all()
    assert ((g - g_ref) == 0).float().mean() > 0.9
    again = gdn.ab_gates(x, w, a_log, dt, hv)
    assert torch.equal(again[0], g) and torch.equal(again[1], beta)


@pytest.mark.parametrize("t", [1, 2, 4, 5, 8, 9, 511, 512, 513, 530])
def test_convolution_around_its_runs_of_tokens(t):
    from deepseek_v4_2080ti_b200.ops import basic
    torch.manual_seed(t)
    c = 264
    x, tail = torch.randn(t, c + 8, device="cuda").bfloat16(), torch.randn(3, c, device="cuda").bfloat16()
    w = torch.randn(c, 4, device="cuda").bfloat16()
    want, new_tail = basic.conv_silu_ref(x[:, :c], w, tail)
    got = basic.conv_silu(x[:, :c], w, tail)
    # one rounding to bf16 and a fast exponential
    assert ((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all() and torch.equal(tail, new_tail)


# the lines between runs of all tokens, of 4, 8 and 16
@pytest.mark.parametrize("t", [3, 6, 7, 191, 192, 193, 196, 200])
def test_convolution_at_the_lines_between_its_runs(t):
    test_convolution_around_its_runs_of_tokens(t)
