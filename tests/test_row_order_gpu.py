"""A 32-bit row is the same number whatever the number of rows beside it, in the kernels over rows by 16-byte pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# widths on both sides of every change of pieces a thread, for few rows and for many; rows that are no whole pieces or too long for them
@pytest.mark.parametrize("D", [30, 64, 256, 260, 516, 1024, 1028, 2048, 2052, 4096, 4100, 8192, 8196])
def test_rows_do_not_depend_on_their_number(D):
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(D)
    R = 300
    a, b, c, d = (torch.randn(R, D, generator=g).cuda() for _ in range(4))
    w, w2 = (1.0 + 0.1 * torch.randn(D, generator=g).cuda() for _ in range(2))

    def all_of(rows):
        x, y, z, u = (t[:rows].contiguous() for t in (a, b, c, d))
        out = [o.rms_scale_add(x, w, 1e-6, 0.7, adds=[z, u]), o.rms_scale_add(x, w, 1e-6, 0.7, adds=[z], second=(y, w2)),
               *o.post_norm_add(x, w, 1e-6, z, scale=0.7, second=(y, -1.3), rounded=torch.bfloat16), o.post_norm_add(x, w, 1e-6, z)[0]]
        if D % 4 == 0 and D <= 8192:       # (element by element the pair of norms has a form for few rows and one for many)
            out += [t for dtype in (torch.float32, torch.bfloat16) for t in o.rms_norm_pair(x, w, w2, 1e-6, dtype)]
        return out

    whole = all_of(R)
    for rows in (1, 63, 64, 299):
        for got, want in zip(all_of(rows), whole):
            assert torch.equal(got, want[:rows]), rows


@pytest.mark.parametrize("D", [4, 64, 128, 132, 256, 260, 384, 512])
def test_many_narrow_rows(D):
    """Several rows a block (the pair of norms from 1,024 rows on), the last block part empty: the rows of a call of few."""
    from gopherllm_b200 import ops as o
    g = torch.Generator().manual_seed(D)
    x, w1, w2 = torch.randn(1027, D, generator=g).cuda(), torch.randn(D, generator=g).cuda(), torch.randn(D, generator=g).cuda()
    for dtype in (torch.float32, torch.bfloat16):
        many = o.rms_norm_pair(x, w1, w2, 1e-6, dtype)
        for at in (0, 500, 1000):
            for few, all_rows in zip(o.rms_norm_pair(x[at:at + 27].contiguous(), w1, w2, 1e-6, dtype), many):
                assert torch.equal(few, all_rows[at:at + 27])
