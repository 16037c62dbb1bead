"""As many rows as an int32 holds: the row counter goes past its end without turning
negative.  (34 GB of input rows; the kernels for patches share the loop's form, but
would take 86 GB.)"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_pack_rows_of_int32_max_rows():
    from mbd_icenav_b200 import sg_ops as ops
    R, ldx = 2 ** 31 - 1, 8
    if torch.cuda.mem_get_info()[0] < R * ldx * 2 + 2 ** 33:
        pytest.skip("the input rows do not fit beside what others hold")
    x = torch.full((R, ldx), 1.0, dtype=torch.bfloat16, device="cuda")
    ops.pack_rows(None, None, x)
    torch.cuda.synchronize()
    rest = sum(int(torch.count_nonzero(part)) for part in x.view(torch.int64).view(-1).split(2 ** 28))
    del x
    torch.cuda.empty_cache()
    assert rest == 0
