"""bench.py's bytes per kernel: the vacuum's row copies are charged to the
kernel that makes them."""
import os
import re

import bench

SRC = os.path.join(os.path.dirname(os.path.abspath(bench.__file__)), "vhlle_b200", "csrc", "vh_step.cu")


def test_the_update_lists_line_is_the_kernels():
    blocks = int(re.search(r"kUpdateMinBlocks = (\d+)", open(SRC).read()).group(1))
    assert bench.UPDATE_LIST_BLOCKS == 148 * blocks


def test_vacuum_copies_are_charged_where_they_are_made():
    prof = {"k_face": (2, 1.0), "k_update": (2, 1.0), "k_visc_prims": (1, 1.0)}
    for cells, copier in ((47 * 61 * 23, "k_update"), (1184 * 128, "k_update"), (1184 * 128 + 1, "k_face"),
                          (101 * 101 * 51, "k_face")):
        none = bench.kernel_alg_bytes(prof, cells, 1, cells)  # matter everywhere
        some = bench.kernel_alg_bytes(prof, cells, 1, cells - 1000)
        listed = {k: bench.KERNEL_BYTES[k][0] * 1000 * prof[k][0] for k in prof}
        for k in prof:
            copies = 1000 * bench.VACUUM_COPY_B * prof[k][0] if k == copier else 0
            assert none[k] - some[k] == listed[k] - copies
        assert bench.kernel_bytes_rule(copier, cells).endswith("x empty cells")
    assert bench.KERNEL_BYTES["k_visc_prims"][0] == 8 * (14 + 8 + 3 + 5 + 9 + 4) + 8
