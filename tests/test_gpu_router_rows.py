"""Router logits of up to 128 tokens: the two fp32 kernels that share this range sum every logit in the same order, so whichever serves a call, a token's logits are the
same bits as in a call of its own. Sizes on both sides of the rule between them (passes over the gate's rows, length of a row) and ragged ones."""
import pytest
import torch

from kyojin_mac_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,H,dtype", [(4, 512, torch.float16), (8, 1024, torch.float16), (16, 1024, torch.bfloat16), (256, 1024, torch.float16), (160, 2048, torch.float16),
                                       (257, 3072, torch.float16), (384, 5120, torch.float16), (512, 4096, torch.float32), (33, 1032, torch.float16), (256, 16384, torch.bfloat16)])
def test_logits_do_not_depend_on_the_number_of_tokens(E, H, dtype):
    g = torch.Generator(device="cuda").manual_seed(E + H)
    x = torch.randn((129, H), device="cuda", generator=g).to(dtype)
    gw, sgw = 0.02 * torch.randn((E, H), device="cuda", generator=g), 0.02 * torch.randn((H,), device="cuda", generator=g)
    alone = torch.cat([ops.router_logits(x[t:t + 1], gw, sgw) for t in range(129)])
    want = x.double() @ torch.cat([gw, sgw[None]]).double().T
    assert ((alone.double() - want).norm() / want.norm()).item() <= 1e-5                    # fp32 sums of up to 16384 products: 2e-7 seen
    for T in (2, 4, 5, 8, 12, 31, 48, 64, 65, 96, 100, 128, 129):
        lg = ops.router_logits(x[:T], gw, sgw)
        assert torch.equal(lg[:, :E + 1], alone[:T, :E + 1]), T
