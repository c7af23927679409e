"""CPU: the three-pass schedule's last pass with the lanes of a tile across the
first digit k1 (adjacent outputs), from the kernel source on the emulator
against the oracle, full tiles and a last tile with lanes missing."""
import numpy as np
import pytest

from conftest import P, rand_field
from test_kernel_emulation import F_LOAD_LF, F_PASS_TW, F_STORE_LF, build_emu, call, root, table


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    return build_emu(tmp_path_factory, ("-DGL_DEVICE_CHECKS",))


@pytest.mark.parametrize("n1,n2,n3,shapes", [(8, 8, 64, [("gen", 8, 1, 1), ("gen", 8, 1, 1), (8, 8, 1)]),
                                             (6, 10, 272, [("gen", 6, 1, 1), ("gen", 10, 1, 1), (16, 17, 1)])])
@pytest.mark.parametrize("inv", [False, True])
def test_rows_across_k1(emu, oracle, n1, n2, n3, shapes, inv):
    n, n23 = n1 * n2 * n3, n2 * n3
    x = rand_field(n, seed=41 + inv)
    s1, out = np.zeros_like(x), np.zeros_like(x)
    w, w23 = root(n, inv), root(n23, inv)
    t1, t2, t3 = (table(root(m, inv), m) for m in (n1, n2, n3))
    lo, hi = table(w, 4096, pow(n, P - 2, P) if inv else 1), table(pow(w, 4096, P), (n + 4095) // 4096)
    lo23, hi23 = table(w23, 4096), table(pow(w23, 4096, P), (n23 + 4095) // 4096)
    flags = F_PASS_TW | F_LOAD_LF | F_STORE_LF
    call(emu, shapes[0], inv, x, s1, 1, n23, 1, n23, n23, flags, t1, t1, lo, hi, unscale=n if inv else 1)
    for k1 in range(n1):
        blk = s1[k1 * n23:(k1 + 1) * n23]
        call(emu, shapes[1], inv, blk, blk, 1, n3, 1, n3, n3, flags, t2, t2, lo23, hi23)
    for k2 in range(n2):  # grid.y of the last pass: row k2 of every block, stored at k1 + n1 k2
        call(emu, shapes[2], inv, s1[k2 * n3:], out[n1 * k2:], n23, 1, 1, n1 * n2, n1, F_STORE_LF, t3, t3)
    assert np.array_equal(out, (oracle.intt if inv else oracle.ntt)(x))
