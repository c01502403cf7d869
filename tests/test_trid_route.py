"""Which Thomas sweep a solve takes, decided on the host (trid_sweep): the split
sweep loads pairs of elements and the on-chip sweep copies rows from 16-byte
boundaries, so an array with another alignment has the streaming sweep, whatever
the context's choice and its size.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include "plc_internal.h"
int main() {
  int nx, nz, split, tile, elem;
  unsigned long long at, smem;
  while (std::scanf("%d %d %d %d %d %llu %llu", &nx, &nz, &split, &tile, &elem, &at, &smem) == 7) {
    plc_ctx c{};
    c.nx = nx;
    c.nz = nz;
    c.trid_split = split;
    c.trid_tile = tile;
    c.trid_smem_max = smem;
    std::printf("%d\n", (int)plc::trid_sweep(&c, elem, reinterpret_cast<const void *>(at)));
  }
}
"""
SPLIT, TILE, STREAM = 0, 1, 2
SMEM = 227 * 1024


@pytest.fixture(scope="module")
def sweeps(tmp_path_factory):
    d = tmp_path_factory.mktemp("trid")
    (d / "route.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT}/include",
                    f"-I{ROOT}/powerllel_channel_sycl_b200/csrc", "-I/usr/local/cuda/include",
                    "-o", d / "route", d / "route.cc"], check=True)

    def run(cases):
        text = "".join(" ".join(str(int(v)) for v in c) + "\n" for c in cases)
        out = subprocess.run([d / "route"], input=text, capture_output=True, text=True, check=True)
        return [int(v) for v in out.stdout.split()]
    return run


def test_unaligned_arrays_stream(sweeps):
    """Every grid, choice and type: one element off a boundary is streamed."""
    cases = [(nx, nz, split, tile, elem, 4096 + 16 * k + elem, SMEM)
             for nx in (12, 32, 64, 768) for nz in (2, 64, 256, 258, 512) for split in (0, 1)
             for tile in (0, 1) for elem in (4, 8) for k in range(3)]
    assert sweeps(cases) == [STREAM] * len(cases)


def test_aligned_arrays(sweeps):
    for elem in (4, 8):
        fits = SMEM // (32 * elem) - 1
        for at in (4096, 4096 + 16):
            assert sweeps([
                (32, 256, 1, 1, elem, at, SMEM),       # split wherever the column fits
                (36, 2, 1, 0, elem, at, SMEM),
                (32, 258, 1, 1, elem, at, SMEM),       # taller: on chip,
                (32, 258, 1, 0, elem, at, SMEM),       # or streamed as tuned,
                (36, 258, 1, 1, elem, at, SMEM),       # in rows of 32 systems,
                (32, fits, 1, 1, elem, at, SMEM),      # within the shared memory
                (32, fits + 2, 1, 1, elem, at, SMEM),
                (32, 64, 0, 1, elem, at, SMEM),        # pinned serial sweeps
                (32, 64, 0, 0, elem, at, SMEM),
            ]) == [SPLIT, SPLIT, TILE, STREAM, STREAM, TILE, STREAM, TILE, STREAM]
    # FP32 pairs lie on 8-byte boundaries; the bulk copies need 16
    assert sweeps([(32, 64, 1, 1, 4, 4104, SMEM), (32, 258, 1, 1, 4, 4104, SMEM),
                   (32, 64, 0, 1, 4, 4104, SMEM)]) == [SPLIT, STREAM, STREAM]
