"""Power-of-two activation scales: the quantiser multiplies by the reciprocal of the scale, which
must give the bytes of the division over the whole exponent range of bf16."""

import pytest
import torch

from moe_bench_b200 import capi
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def ue8m0():
    capi.set_fp8_scale_format("ue8m0")
    yield
    capi.use_reference_fp8_scale_format()


@pytest.mark.parametrize("rows,offset", [(1, 0), (301, 0), (301, 8)])
def test_every_binade_matches_the_division(ue8m0, rows, offset):
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, 512, generator=gen)
    exponent = torch.randint(-38, 120, (rows, 4), generator=gen).float().repeat_interleave(128, 1)
    x = (x * torch.exp2(exponent)).to(torch.bfloat16)
    x[0, :128] = 0
    x[0, 128:256] = 448.0                      # amax / 448 a power of two already
    x[0, 256:384] = -448.0 * 2.0**20
    x[0, 300] = 3.0e38                         # the other elements fall below the smallest e4m3 value
    oq, os_ = O.group_quant_fp8(x, scale_format="ue8m0")
    if offset:  # the e4m3 buffer of a caller of the C ABI may be 8-byte aligned only
        raw = torch.zeros(rows * 512 + 16, dtype=torch.uint8, device=DEV)
        shift = (-raw.data_ptr()) % 16 + offset
        q = raw[shift : shift + rows * 512].view(rows, 512)
        s = torch.empty(rows, 4, device=DEV)
        xd = x.to(DEV)
        rc = capi.load().mb200_group_quant_fp8(xd.data_ptr(), rows, 512, q.data_ptr(), s.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    else:
        q, s = capi.group_quant_fp8(x.to(DEV))
    assert torch.equal(s.cpu(), os_)
    assert torch.equal(q.cpu().view(torch.uint8), oq.view(torch.uint8))
