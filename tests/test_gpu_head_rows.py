"""The head's encoder rows in the forms that users hold them in: other integer types,
strided, and activations that do not begin on a 16-byte boundary; shared by few rows
(one product for them) and not."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [10, 13])  # three encoder rows: packed beside every row, and shared
def test_head_takes_encoder_rows_in_any_form(R):
    from mbd_icenav_b200.surrogate import SurrogateNet, enc_dim
    net = SurrogateNet(horizon=16, device="cuda", seed=1)
    g = torch.Generator().manual_seed(R)
    E, P = enc_dim(), 3
    enc = torch.randn((P, E), generator=g).to(torch.bfloat16).cuda()
    extra = torch.randn((R, net.n_extra), generator=g).cuda()
    row = torch.randint(0, P, (R,), generator=g, dtype=torch.int32).cuda()
    want = net.head(enc, extra, enc_row=row).clone()
    off = torch.empty(P * E + 1, dtype=torch.bfloat16, device="cuda")[1:].view(P, E)
    off.copy_(enc)
    wide = torch.empty((P, E + 1), dtype=torch.bfloat16, device="cuda")[:, :E]
    wide.copy_(enc)
    for e in (off, wide):
        assert torch.equal(net.head(e, extra, enc_row=row), want)
    for r in (row.long(), torch.stack([row, 2 - row], 1)[:, 0]):
        assert torch.equal(net.head(enc, extra, enc_row=r), want)
    one = net.head(enc[:1], extra, enc_row=torch.zeros(R, dtype=torch.int32, device="cuda")).clone()
    assert torch.equal(net.head(enc[:1], extra, enc_row=torch.zeros(1, dtype=torch.int64, device="cuda").expand(R)), one)
    torch.cuda.synchronize()
