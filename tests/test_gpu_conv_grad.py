"""The weight-gradient kernel at the sizes where its split can go wrong: the
edges of its 64-pixel columns, images of one row, fewer rows than blocks, a
block that ends inside one column and starts in the next, one block for all.

The reference is torch's FP64 gradient of the same BF16 inputs.  Their products
are exact in FP32.  A block adds two products of 16 pixels per row it marches to
each of its accumulators, and a tensor-core addition may cut off up to 2^-23 of the
running sum, half of that on average: steps * 2^-23 for the rows of one block.  The
additions after that (two accumulators, the blocks in eight chains) round to
nearest: 2 + 3 + 19 + 8 of them at 2^-24 each are 2e-6.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("n,h,w,nparts", [
    (1, 1, 1, 1), (1, 1, 64, 3), (2, 2, 65, 7), (3, 5, 63, 400), (1, 37, 130, 11), (2, 90, 129, 1), (5, 33, 128, 304),
])
def test_weight_grad_splits(tl, built_lib, cin, cout, n, h, w, nparts):
    gen = torch.Generator().manual_seed(n * 1000 + h * 10 + w + cin)
    x = torch.randn(n, h, w, cin, generator=gen).to(torch.bfloat16)
    dz = torch.randn(n, h, w, cout, generator=gen).to(torch.bfloat16)
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    dw = torch.stack([torch.einsum("nhwo,nhwi->oi", dz.double(), xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w])
                      for t in range(9)], dim=1)
    ref = torch.cat([dw.reshape(-1), dz.double().sum(dim=(0, 1, 2))])
    lib, xd, zd = tl._abi.load(), x.cuda(), dz.cuda()
    nw = ref.numel()
    parts = torch.full((nparts * nw,), float("nan"), device="cuda")
    got = []
    for _ in range(2):
        out = torch.full((nw,), float("nan"), device="cuda")
        rc = lib.tl_conv3x3_weight_grad(xd.data_ptr(), zd.data_ptr(), parts.data_ptr(), nparts, out.data_ptr(), n, h,
                                        w, cin, cout, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        got.append(out.cpu())
    assert torch.equal(got[0], got[1])
    blocks = min(nparts, torch.cuda.get_device_properties(0).multi_processor_count)
    steps = -(-n * -(-w // 64) * h // blocks)
    assert torch.linalg.norm(got[0].double() - ref) <= (2e-6 + steps * 2.0 ** -23) * torch.linalg.norm(ref)
