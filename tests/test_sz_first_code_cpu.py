"""Tiles whose values lie so far from 0, in steps of the grid, that they have no codes: which first codes the packer takes
(csrc/kernels/ccb_sz_layout.h), for every sum that it can form, and what the host codec makes of such a tile."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from ccbench_b200.ops import sz


def test_first_codes_are_told_apart_for_every_sum(tmp_path):
    if not shutil.which("gcc"):
        pytest.skip("no C compiler")
    src = tmp_path / "t.c"
    src.write_text(r'''
#include <string.h>
#include "ccb_sz_layout.h"
int main(void) {
    const float magic = 12582912.f;
    uint32_t zero, bits = 0;
    memcpy(&zero, &magic, 4);
    do {   /* every float, NaN and infinities too: near is what is a whole number of steps, at most that many */
        float r;
        memcpy(&r, &bits, 4);
        const double code = (double)r - 12582912.0;
        for (uint32_t most = 31999; most < 3000000; most += 2061057)   /* 31999 and 2^21 - 4096 */
            if (ccb_sz_code_within(bits - zero, most) != (code >= -(double)most && code <= (double)most)) return 1;
    } while (++bits);
    return ccb_sz_code_within(0x80000000u, (1u << 21) - 4096) ? 2 : 0;
}''')
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["gcc", "-O2", "-I" + os.path.join(root, "csrc", "kernels"), str(src), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


@pytest.mark.parametrize("value,eb", [(-50282496.0, 1.0), (-5028.2495, 1e-4)])
def test_a_value_of_no_code_is_kept_as_it_is(value, eb):
    field = np.full((8, 8, 32), value, np.float32)
    assert (sz.decode_cpu(sz.encode_cpu(field, eb)) == field).all()
