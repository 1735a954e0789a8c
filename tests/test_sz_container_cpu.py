"""The self-describing container of the error-bounded codec: pure tensor code, testable
without a GPU on a made-up buffer of group slots."""
import pytest
import torch

from ccbench_b200.ops import sz


def _fake_slots(shape, seed=0):
    ngroups = sz.capacity(shape) // sz.GROUP_STRIDE
    g = torch.Generator().manual_seed(seed)
    buf = torch.randint(0, 256, (ngroups, sz.GROUP_STRIDE), dtype=torch.uint8, generator=g)
    sizes = torch.randint(4, 500, (ngroups, 8), dtype=torch.int32, generator=g) * 16
    buf[:, :sz.GROUP_HEADER] = sizes.view(torch.uint8).reshape(ngroups, sz.GROUP_HEADER)
    return buf.view(-1), sizes


def test_roundtrip_keeps_exactly_the_used_bytes():
    shape = (40, 24, 100)
    buf, sizes = _fake_slots(shape)
    blob = sz.to_container(buf, shape, 1e-3)
    ngroups = sizes.shape[0]
    assert blob.numel() == sz.HEADER_BYTES + 4 * ngroups + int(sizes.sum()) + ngroups * sz.GROUP_HEADER
    back, shape2, eb = sz.from_container(blob)
    assert tuple(shape2) == shape and abs(eb - 1e-3) < 1e-9
    a, b = buf.view(ngroups, -1), back.view(ngroups, -1)
    for gi in range(ngroups):
        used = sz.GROUP_HEADER + int(sizes[gi].sum())
        assert torch.equal(a[gi, :used], b[gi, :used])
        assert int(b[gi, used:].max()) == 0


def test_damaged_containers_are_refused():
    shape = (16, 16, 64)
    buf, _ = _fake_slots(shape, 1)
    blob = sz.to_container(buf, shape, 1e-2)
    for cut in (blob[:-5], torch.cat([blob, blob[:3]])):
        with pytest.raises(ValueError):
            sz.from_container(cut)
    wrong = blob.clone()
    wrong[4] = 9   # version
    with pytest.raises(ValueError):
        sz.from_container(wrong)


def test_cpu_codec_round_trip_matches_the_restatement():
    import numpy as np

    rng = np.random.default_rng(0)
    zz, yy, xx = np.meshgrid(np.arange(20), np.arange(13), np.arange(70), indexing="ij")
    field = (np.sin(zz / 5.0) * np.cos(yy / 3.0) + 0.01 * xx + 1e-3 * rng.standard_normal(zz.shape)).astype(np.float32)
    eb = 1e-3
    blob = sz.encode_cpu(field, eb)
    recon, nbytes = sz.restate(field, eb)
    back = sz.decode_cpu(blob)
    assert back.shape == field.shape and np.array_equal(back, recon)
    assert float(np.abs(back - field).max()) <= np.float32(eb)
    ngroups = sz.capacity(field.shape) // sz.GROUP_STRIDE
    assert blob.size == sz.HEADER_BYTES + 4 * ngroups + nbytes + ngroups * sz.GROUP_HEADER
    # the tensor-side container reader accepts what the CPU encoder wrote
    buf, shape, eb2 = sz.from_container(torch.from_numpy(blob))
    assert tuple(shape) == field.shape and abs(eb2 - eb) < 1e-9
    assert np.array_equal(sz.decode_cpu(sz.to_container(buf, shape, eb2).numpy()), recon)


def test_cpu_codec_stores_unquantisable_tiles_raw():
    import numpy as np

    field = np.zeros((8, 8, 64), dtype=np.float32)
    field[:, :, :32] = np.linspace(-1, 1, 8 * 8 * 32, dtype=np.float32).reshape(8, 8, 32)
    field[3, 4, 40] = np.nan
    field[1, 1, 50] = 3e30
    blob = sz.encode_cpu(field, 1e-3)
    back = sz.decode_cpu(blob)
    assert np.array_equal(back[:, :, 32:], field[:, :, 32:], equal_nan=True)     # raw tile: bit exact
    assert float(np.abs(back[:, :, :32] - field[:, :, :32]).max()) <= np.float32(1e-3)


@pytest.mark.parametrize("tile,size", [(0, 1 << 20), (2, 8272), (3, 20), (7, -16), (5, 48)])
def test_tile_sizes_that_cannot_be_are_refused(tile, size):
    """A flipped word inside the payload, with the list of group sizes intact."""
    buf, sizes = _fake_slots((40, 24, 100))
    blob = sz.to_container(buf, (40, 24, 100), 1e-3)
    ngroups = sizes.shape[0]
    at = sz.HEADER_BYTES + 4 * ngroups + sz.GROUP_HEADER + int(sizes[0].sum()) + 4 * tile   # group 1
    bad = blob.clone()
    bad[at:at + 4].view(torch.int32).fill_(size)
    with pytest.raises(ValueError):
        sz.from_container(bad)
    with pytest.raises(ValueError):
        sz.decode_cpu(bad.numpy())
    slots = buf.clone()
    slots[sz.GROUP_STRIDE + 4 * tile:sz.GROUP_STRIDE + 4 * tile + 4].view(torch.int32).fill_(size)
    with pytest.raises(ValueError):
        sz.to_container(slots, (40, 24, 100), 1e-3)


def test_tile_sizes_that_do_not_make_their_group_are_refused():
    buf, sizes = _fake_slots((40, 24, 100))
    blob = sz.to_container(buf, (40, 24, 100), 1e-3)
    at = sz.HEADER_BYTES + 4 * sizes.shape[0] + 8
    blob[at:at + 4].view(torch.int32).fill_(int(sizes[0, 2]) + (16 if int(sizes[0, 2]) < 8000 else -16))
    with pytest.raises(ValueError):
        sz.from_container(blob)


def test_row_widths_that_cannot_be_are_refused_by_the_host_decoder():
    import numpy as np

    blob = sz.encode_cpu(np.linspace(0, 1, 8 * 8 * 32, dtype=np.float32).reshape(8, 8, 32), 1e-3)
    blob[sz.HEADER_BYTES + 4 + sz.GROUP_HEADER + 9] = 33
    with pytest.raises(ValueError):
        sz.decode_cpu(blob)


def test_a_tile_that_passes_the_layouts_checks_lies_inside_its_slot(tmp_path):
    """csrc/kernels/ccb_sz_layout.h, which the kernels read buffers by: every offset a sum of size words
    can give, and every width byte in each place of its word."""
    import os
    import shutil
    import subprocess

    if not shutil.which("gcc"):
        pytest.skip("no C compiler")
    src = tmp_path / "t.c"
    src.write_text(r'''
#include "ccb_sz_layout.h"
int main(void) {
    for (unsigned k = 0; k < CCB_SZ_TILES; ++k)
        for (uint64_t off = 0; off < (1ull << 32); off += off < (1u << 18) ? 1 : 4093)
            if (ccb_sz_offset_ok((uint32_t)off, k) && (off % 16 || CCB_SZ_GROUP_HEADER + off + CCB_SZ_TILE_CAP > CCB_SZ_GROUP_STRIDE)) return 1;
    if (!ccb_sz_offset_ok(7 * CCB_SZ_TILE_CAP, 7) || !ccb_sz_offset_ok(0, 0)) return 2;   /* raw tiles only */
    for (int at = 0; at < 4; ++at)
        for (unsigned b = 0; b < 256; ++b)
            for (unsigned other = 0; other < 256; other += 17)
                if (ccb_sz_widths_ok((other * 0x01010101u & ~(0xffu << 8 * at)) | b << 8 * at) != (b <= 32 && other <= 32)) return 3;
    if (CCB_SZ_ROWS + 4 * CCB_SZ_ROWS * 32 != CCB_SZ_TILE_CAP) return 4;   /* what widths of 32 add up to */
    for (uint32_t s = 0; s < 70000; ++s)
        if (ccb_sz_size_ok(s) != (s == 0 || (s % 16 == 0 && s >= 64 && s <= 8256))) return 5;
    return ccb_sz_size_ok(0xfffffff0u) ? 6 : 0;
}''')
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["gcc", "-O2", "-I" + os.path.join(root, "csrc", "kernels"), str(src), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0
