"""Which Thomas sweep a solve takes, decided on the host (trid_sweep): the split
sweep loads pairs of elements and the on-chip sweep copies rows from 16-byte
boundaries, so an array with another alignment has the streaming sweep, whatever
the context's choice and its size; and the grids whose columns the split sweep
takes unless it is pinned.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include "plc_internal.h"
int main() {
  int nx, ny, nz, split, tile, pinned, elem;
  unsigned long long at, smem;
  while (std::scanf("%d %d %d %d %d %d %d %llu %llu", &nx, &ny, &nz, &split, &tile, &pinned, &elem,
                    &at, &smem) == 9) {
    plc_ctx c{};
    c.nx = nx;
    c.ny = ny;
    c.nz = nz;
    c.device_sms = 148;
    c.trid_pinned = pinned;
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
    cases = [(nx, 24, nz, split, tile, pin, elem, 4096 + 16 * k + elem, SMEM)
             for nx in (12, 32, 64, 768) for nz in (2, 64, 256, 258, 512) for split in (0, 1)
             for tile in (0, 1) for pin in (0, 1) for elem in (4, 8) for k in range(3)]
    assert sweeps(cases) == [STREAM] * len(cases)


def test_aligned_arrays(sweeps):
    for elem in (4, 8):
        fits = SMEM // (32 * elem) - 1
        for at in (4096, 4096 + 16):
            for pin in (0, 1):
                assert sweeps([
                    (32, 24, 256, 1, 1, pin, elem, at, SMEM),       # split wherever the column fits
                    (36, 24, 2, 1, 0, pin, elem, at, SMEM),
                    (32, 24, 258, 1, 1, pin, elem, at, SMEM),       # taller: on chip,
                    (32, 24, 258, 1, 0, pin, elem, at, SMEM),       # or streamed as tuned,
                    (36, 24, 258, 1, 1, pin, elem, at, SMEM),       # in rows of 32 systems,
                    (32, 24, fits, 1, 1, pin, elem, at, SMEM),      # within the shared memory
                    (32, 24, fits + 2, 1, 1, pin, elem, at, SMEM),
                    (32, 24, 64, 0, 1, pin, elem, at, SMEM),        # serial sweeps
                    (32, 24, 64, 0, 0, pin, elem, at, SMEM),
                ]) == [SPLIT, SPLIT, TILE, STREAM, STREAM, TILE, STREAM, TILE, STREAM]
    # FP32 pairs lie on 8-byte boundaries; the bulk copies need 16
    assert sweeps([(32, 24, 64, 1, 1, 0, 4, 4104, SMEM), (32, 24, 258, 1, 1, 0, 4, 4104, SMEM),
                   (32, 24, 64, 0, 1, 0, 4, 4104, SMEM)]) == [SPLIT, STREAM, STREAM]


# grid, and whether the FP64 and the mixed form take the split sweep on 148 SMs
RULE = [((32, 24, 16), True, True), ((64, 48, 48), True, True), ((162, 108, 90), True, True),
        ((128, 96, 2), True, True), ((192, 144, 18), False, True), ((384, 192, 18), False, False),
        ((512, 288, 24), False, False), ((512, 288, 26), False, True), ((192, 144, 30), False, True),
        ((256, 128, 32), True, True), ((216, 192, 38), True, True), ((256, 192, 38), False, True),
        ((256, 192, 130), False, True), ((512, 288, 216), False, True), ((512, 288, 218), True, True),
        ((512, 384, 130), False, False), ((512, 384, 54), False, True), ((512, 384, 56), True, True),
        ((768, 384, 108), False, True), ((768, 384, 110), True, True), ((768, 384, 130), False, False),
        ((768, 384, 250), True, False), ((1024, 512, 66), False, False),
        ((1024, 512, 126), True, False)] + [((nx, nx // 2, nz), True, True)
                                             for nx in (64, 768, 1536) for nz in (64, 128, 256)]


def test_split_sweep_where_it_pays(sweeps):
    for q, elem in enumerate((8, 4)):
        assert sweeps([(*g, 1, 0, 0, elem, 4096, SMEM) for g, *_ in RULE]) == \
            [SPLIT if r[q] else STREAM for _, *r in RULE]
        # pinned, wherever the column fits
        assert sweeps([(*g, 1, 0, 1, elem, 4096, SMEM) for g, *_ in RULE]) == [SPLIT] * len(RULE)
