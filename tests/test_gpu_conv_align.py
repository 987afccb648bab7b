"""Forward and input gradient with outputs on 32-byte boundaries (whole sectors
at a time) and 16 bytes off them: the same bytes."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (2, 5, 127), (1, 19, 129), (3, 33, 260)])
def test_output_alignment(tl, built_lib, cin, cout, mode, n, h, w):
    gen = torch.Generator().manual_seed(n * 1000 + h * 10 + w + cin)
    rnd = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16).cuda()
    x, wt, gz0 = rnd(n, h, w, cin), rnd(cout * 9 * cin), rnd(n * h * w * cout)
    bias = torch.randn(cout, generator=gen).cuda()
    lib, st = tl._abi.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = []
    for off in (0, 8):  # elements of two bytes
        gz, z, out = (torch.zeros(gz0.numel() + 16, dtype=torch.bfloat16, device="cuda") for _ in range(3))
        gz[off:off + gz0.numel()] = gz0
        p = lambda t: t.data_ptr() + 2 * off
        rc = lib.tl_conv3x3_forward(x.data_ptr(), wt.data_ptr(), bias.data_ptr(), p(gz) if mode == 2 else None,
                                    p(z) if mode == 1 else None, p(out), None, n, h, w, cin, cout, mode, st)
        assert rc == 0
        got.append((z[off:off + gz0.numel()].cpu(), out[off:off + gz0.numel()].cpu(), out[off + gz0.numel():].cpu()))
    for a, b in zip(got[0][:2], got[1][:2]):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert not got[0][2].any() and not got[1][2][:8].any()
