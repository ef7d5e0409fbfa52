"""Rules that keep a product on the group tiles within what their kernels can
hold (panel_limits.cuh), compiled as plain C++: no GPU, and no matrix of that
size, is needed."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "panel_limits.cuh"
int main(int argc, char** argv) {
  long long v[8] = {};
  for (int i = 2; i < argc; ++i) v[i - 2] = atoll(argv[i]);
  bool ok = false;
  if (!strcmp(argv[1], "blocks")) ok = lamb::panel_blocks_ok(v[0], v[1], v[2]);
  if (!strcmp(argv[1], "atoms")) ok = lamb::panel_atoms_ok(v[0], v[1], v[2]);
  if (!strcmp(argv[1], "norms")) ok = lamb::norm_index_ok(v[0], v[1]);
  printf("%d\n", ok);
  return 0;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("limits")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "limits")
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(REPO, "lamb_b200", "csrc"),
                           str(d / "main.cpp"), "-o", exe])
    return lambda name, *v: subprocess.check_output([exe, name, *map(str, v)], text=True).strip() == "1"


def test_block_counts_fit_the_kernel_s_32_bits(rule):
    """The kernel's block index is int: row_p[row] + blocks before the column."""
    top = 2 ** 31 - 1
    assert rule("blocks", top, top, top)
    for at in range(3):
        v = [1000] * 3
        v[at] = top + 1
        assert not rule("blocks", *v)
    # 51,200 atoms of one row, 5 % structured fill in A and B: C has every block
    assert not rule("blocks", 131072000, 131072000, 51200 * 51200)


def test_block_norms_have_32_bit_indices(rule):
    top = 2 ** 31 - 1
    assert rule("norms", top, 1) and rule("norms", top + 1, 0)
    assert not rule("norms", top + 1, 1)


@pytest.mark.parametrize("at,top", [(0, 262144), (1, 65536), (2, 51200)])
def test_atoms_by_role(rule, at, top):
    v = [100] * 3
    v[at] = top
    assert rule("atoms", *v)
    v[at] = top + 1
    assert not rule("atoms", *v)
    v[at] = 0
    assert not rule("atoms", *v)


def test_masks_of_a_super_row_fit_shared_memory(rule):
    """Two column groups take 8 bytes, every atom may be a group; 227 KB less the
    block reduction's storage is what one CTA has."""
    lo, hi = 1, 1 << 20  # the first is taken, the second is not
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if rule("atoms", 1, 1, mid) else (lo, mid)
    assert 8 * ((lo + 1) // 2) + 4096 <= 232448
