"""The error-bounded codec where its accesses to a field change: lines on 32 bytes, on 16 and anywhere
(extents and a start of the buffer that allow no wider), tiles cut off in each direction, and packed
tiles from a few bytes to more than a warp stages (4 KiB), against the host codec byte for byte."""
import numpy as np
import pytest
import torch

from ccbench_b200.ops import sz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 10, 40), (8, 8, 36), (17, 3, 33), (1, 1, 1), (3, 70, 31), (20, 16, 264)])
@pytest.mark.parametrize("start", [0, 4, 1])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 400.0, 1e5])   # widths of none, about 8, 16 and 24 bits at a bound of 1e-2
def test_bytes_and_values_at_every_line_width(shape, start, scale):
    n = int(np.prod(shape))
    host = torch.randn(n, generator=torch.Generator().manual_seed(n + start)) * scale
    field = torch.empty(n + start, device="cuda")[start:].copy_(host).view(shape)
    eb = 1e-2
    buf, used = sz.compress(field, eb)
    want = sz.encode_cpu(host.view(shape).numpy(), eb)
    assert np.array_equal(sz.to_container(buf, shape, eb).cpu().numpy(), want)
    assert int(used) == want.size - sz.HEADER_BYTES - 4 * (buf.numel() // sz.GROUP_STRIDE) - sz.GROUP_HEADER * (buf.numel() // sz.GROUP_STRIDE)
    out = torch.full((n + start + 8,), 7.0, device="cuda")
    target = out[start:start + n]
    sz._check(sz._decl().ccb_sz_decompress(buf.data_ptr(), shape[2], shape[1], shape[0], eb, target.data_ptr(), sz._stream()))
    torch.cuda.synchronize()
    assert np.array_equal(target.view(shape).cpu().numpy(), sz.decode_cpu(want))
    assert (out[:start] == 7).all() and (out[start + n:] == 7).all()


@pytest.mark.parametrize("damage", ["none", "short", "groups", "size", "payload", "magic"])
def test_container_opened_on_the_device(damage):
    shape, eb = (20, 30, 70), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda()
    buf, _ = sz.compress(field, eb)
    blob = sz.to_container(buf, shape, eb)
    words = blob[:sz.HEADER_BYTES + 8].view(torch.int32)
    if damage == "short":
        blob = blob[:sz.HEADER_BYTES + 60].clone()
    elif damage == "groups":      # more than the blob has room for
        words[7] = 1 << 30
    elif damage == "size":        # of the first group
        words[10] += 4
    elif damage == "payload":
        blob = blob[:-4].clone()
    elif damage == "magic":
        words[0] += 1
    if damage == "none":
        back, got_shape, got_eb = sz.from_container(blob)
        assert got_shape == shape and abs(got_eb - eb) < 1e-9
        assert torch.equal(sz.decompress(back, shape, got_eb), sz.decompress(buf, shape, eb))
        assert torch.equal(sz.to_container(back, shape, eb), blob)
    else:
        with pytest.raises(ValueError):
            sz.from_container(blob)


@pytest.mark.parametrize("start", [4, 8, 16])
def test_packed_and_raw_tiles_from_a_buffer_on_four_bytes(start):
    shape, eb = (17, 20, 96), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(2))
    field[:8, :8, 32:64] = 1e30
    buf, _ = sz.compress(field.cuda(), eb)
    moved = torch.empty(buf.numel() + start, dtype=torch.uint8, device="cuda")[start:]
    moved.copy_(buf)
    assert torch.equal(sz.decompress(moved, shape, eb), sz.decompress(buf, shape, eb))
