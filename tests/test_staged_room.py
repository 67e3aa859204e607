"""CPU tests: the rooms of the staged encode's per-launch state for launches
far larger than a test can run, from its own sizing functions compiled for the
host."""

import subprocess

import pytest

from nebc7_gb300 import _native

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "bc7_staged.cuh"
int main(int argc, char** argv)
{
	using namespace nebc7;
	for (int i = 1; i < argc; i++)
	{
		const int n = atoi(argv[i]);
		const Stages s = SplitStaged((uint8_t*)0x10000, n, false);
		printf("%d %d %d %d %zu %zu\n", n, s.impCap, s.laterCap, s.handedCap, StagedScratchBytes(n), sizeof(SplitResult));
	}
	return 0;
}
"""

SIZES = [1, 1000, 43_000, 65_536, 1 << 20, 5_591_000, 5_592_000, 1 << 23, 1 << 24, 1 << 28]


@pytest.fixture(scope="module")
def rooms(tmp_path_factory):
    d = tmp_path_factory.mktemp("rooms")
    (d / "rooms.cu").write_text(PROGRAM)
    subprocess.run([_native.nvcc(), *_native.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(_native.CSRC),
                    str(d / "rooms.cu"), "-o", str(d / "rooms")], check=True)
    out = subprocess.run([str(d / "rooms"), *map(str, SIZES)], check=True, capture_output=True, text=True).stdout
    return {int(l.split()[0]): [int(v) for v in l.split()[1:]] for l in out.splitlines()}


@pytest.mark.parametrize("n", SIZES)
def test_kept_results_fit_their_field(rooms, n):
    """A kept result's slot shares a 32-bit word with its candidate (up to 63):
    24 bits, all ones for "not kept"."""
    results = rooms[n][0]
    assert results == min(3 * n + 1024, n + 2 ** 17, 0xFFFFFF)
    for slot in (0, results - 1):
        word = (63 << 24) | slot
        assert (word >> 24, word & 0xFFFFFF) == (63, slot) and slot != 0xFFFFFF and word < 0x7FFFFFFF
    assert rooms[n][3] >= n * (96 + 6 * 4) + results * rooms[n][4]


@pytest.mark.parametrize("n", SIZES)
def test_state_bytes(rooms, n):
    """The bound the header gives, and later rounds whose tasks (64 a block) an
    int can number."""
    results, later, handed, total, _ = rooms[n]
    assert total <= 172 * n + 14_000_000
    assert handed == min(n, 2048) and later >= min(n, 1 << 24) and later * 64 <= 2 ** 30
