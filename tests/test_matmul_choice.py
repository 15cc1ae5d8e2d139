"""Which kernel takes a product: the rule is host arithmetic, compiled here by itself."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hologram_b200", "csrc")
TILE, WALK, PAIRS, HALVES = range(4)
SHIM = """
#include "gemm_choice.h"
extern "C" int choose(unsigned sms, unsigned m, unsigned k, unsigned n, int linear, unsigned* slices) {
    int bn;
    const unsigned kblocks = (k + BK - 1) / BK;
    if (linear) linear_tile_choice(sms, m, n, kblocks, &bn, slices);
    else tile_choice(sms, m, n, kblocks, &bn, slices);
    return big_choice(sms, m, n, kblocks, linear ? *slices : 1);
}
"""


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("choice")
    (d / "choice.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "choice.so"), str(d / "choice.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "choice.so"))

    def call(m, k, n, linear=True):
        slices = ctypes.c_uint32()
        return lib.choose(148, m, k, n, int(linear), ctypes.byref(slices)), slices.value
    return call


@pytest.mark.parametrize("m,k,n,slices", [(256, 10240, 2048, 2), (256, 8192, 2048, 2), (200, 8192, 512, 8), (130, 10240, 200, 8), (1024, 2048, 64, 8), (1536, 8192, 128, 6), (2048, 10240, 64, 8)])
def test_products_that_split_k_keep_their_slices(choose, m, k, n, slices):
    # on pairs 256 x 8192 x 512 took 34 us, in eight slices 13: the estimate must know of the slices
    assert choose(m, k, n) == (TILE, slices)


@pytest.mark.parametrize("m,k,n,linear,kernel", [
    (256, 512, 2048, True, HALVES),      # two slices of four k-blocks: the sum of 64 rows a CTA costs more than the pair (15 us, 8.6)
    (1024, 8192, 2048, True, HALVES), (1024, 2048, 1344, True, HALVES), (256, 8192, 512, False, HALVES),      # a matmul does not split these
    (4096, 4096, 4096, False, PAIRS), (2048, 10240, 2048, True, PAIRS), (292, 2048, 512, False, TILE), (128, 8192, 8192, True, TILE)])
def test_other_products_keep_their_kernel(choose, m, k, n, linear, kernel):
    assert choose(m, k, n, linear)[0] == kernel


@pytest.mark.parametrize("name,kernel", [("tile", TILE), ("walk", WALK), ("pairs", PAIRS), ("halves", HALVES)])
def test_a_kernel_can_be_named(choose, monkeypatch, name, kernel):
    monkeypatch.setenv("HOLO_GEMM_KERNEL", name)
    assert choose(129, 512, 128)[0] == kernel and choose(4096, 4096, 4096)[0] == kernel
    assert choose(128, 4096, 4096)[0] == TILE      # one row tile always takes a CTA per tile
