"""The weight gradient on either side of the line from which two blocks run on an
SM (16 rows of 64 pixels an SM), up to blocks that march long enough for their
rings of rows to turn many times, with as many partials as blocks and more.

Reference and error model as in test_gpu_conv_grad.py: rows * 2^-23 for the rows
that one block marches; the additions after that, the blocks' partials in eight
chains among them (2 + 3 + 38 + 8 for 304 blocks), 51 * 2^-24 = 3.1e-6.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("n,h,w,per_sm", [
    (1, -1, 64, 2), (1, 0, 64, 2), (1, 1, 64, 3),  # h: rows an SM times SMs, and this many more
    (7, 131, 200, 2), (32, 128, 128, 2), (3, 511, 255, 1),
])
def test_weight_grad_blocks(tl, built_lib, cin, cout, n, h, w, per_sm):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h = 16 * sms + h if h < 2 else h
    nparts = per_sm * sms
    gen = torch.Generator().manual_seed(n * 1000 + h * 10 + w + cin)
    x = torch.randn(n, h, w, cin, generator=gen).to(torch.bfloat16).cuda()
    dz = torch.randn(n, h, w, cout, generator=gen).to(torch.bfloat16).cuda()
    xp, zd = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1)), dz.double().reshape(-1, cout)
    dw = torch.stack([zd.T @ xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin) for t in range(9)], dim=1)
    ref = torch.cat([dw.reshape(-1), zd.sum(dim=0)])
    nw = ref.numel()
    lib = tl._abi.load()
    parts = torch.full((nparts * nw,), float("nan"), device="cuda")
    got = []
    for _ in range(2):
        out = torch.full((nw,), float("nan"), device="cuda")
        rc = lib.tl_conv3x3_weight_grad(x.data_ptr(), dz.data_ptr(), parts.data_ptr(), nparts, out.data_ptr(), n, h, w,
                                        cin, cout, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        got.append(out)
    assert torch.equal(got[0], got[1])
    rows = n * -(-w // 64) * h
    blocks = min(nparts, (2 if rows >= 16 * sms else 1) * sms)
    bound = 3.1e-6 + -(-rows // blocks) * 2.0 ** -23
    assert torch.linalg.norm(got[0].double() - ref) <= bound * torch.linalg.norm(ref)
