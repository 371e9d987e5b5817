"""3x3x3 convolution at the edges of its tiles: depth and height 1, output-line
blocks that end early (blocks of 4 and 2 lines), every channel pair.  Inputs,
weights and biases are small whole numbers, so every FP32 sum is exact in any
order (|sum| <= 27 x 96 x 64 < 2^24) and the output is the whole number rounded
once to BF16: compared for equality."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

PAIRS = [(16, 16), (16, 32), (16, 48), (32, 16), (32, 32), (32, 64), (32, 96), (48, 16), (64, 32),
         (64, 64), (96, 32)]


@pytest.mark.parametrize("cin,cout", PAIRS)
@pytest.mark.parametrize("D,H,W", [(1, 1, 128), (1, 2, 256), (2, 3, 128), (2, 4, 128), (1, 9, 128)])
def test_conv_edges(cin, cout, D, H, W):
    import torch
    import torch.nn.functional as F
    from hrdayapy_b200 import _lib
    from hrdayapy_b200.convref import pack_weights
    g = torch.Generator().manual_seed(100 * cin + cout + H)
    x = torch.randint(-8, 9, (D, H, W, cin), generator=g).to(torch.bfloat16)
    w = torch.randint(-8, 9, (cout, cin, 3, 3, 3), generator=g).to(torch.bfloat16)
    b = torch.randint(-8, 9, (cout,), generator=g).float()
    ref = F.conv3d(x.double().permute(3, 0, 1, 2)[None], w.double(), padding=1)[0]
    ref = (ref.permute(1, 2, 3, 0) + b.double()).float().to(torch.bfloat16)
    dev = torch.device("cuda")
    xd, bd = x.to(dev).contiguous(), b.to(dev).contiguous()
    wp = torch.from_numpy(pack_weights(w.float().numpy())).to(torch.bfloat16).to(dev).contiguous()
    yd = torch.empty(D, H, W, cout, dtype=torch.bfloat16, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    p = [C.c_void_p(t.data_ptr()) for t in (xd, wp, bd, yd)]
    _lib.check(_lib.lib().hp_conv3_forward(*p, None, D, H, W, cin, cout, 1,
                                           C.c_void_p(err.data_ptr()), None), "hp_conv3_forward")
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(yd.cpu(), ref)
