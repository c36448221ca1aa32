"""The rules that pick an expert GEMM kernel from sizes, compiled for the host, against the calls they were measured on."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("choice") / "libchoiceprobe.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(ROOT, "tests", "kernel_choice_probe.cpp"), "-o", str(so)])
    return C.CDLL(str(so))


# rows, experts, d, F, shared expert, us of the integer-MMA kernel, us of the widening kernel
I8 = [(130, 8, 4096, 14336, 0, 267, 377), (192, 8, 4096, 14336, 0, 284, 379), (256, 8, 4096, 14336, 0, 319, 389),
      (192, 16, 4096, 7168, 0, 280, 380), (160, 4, 4096, 14336, 0, 271, 280), (224, 4, 4096, 14336, 0, 219, 284),
      (192, 3, 4096, 14336, 0, 267, 243), (250, 3, 4096, 14336, 0, 292, 247), (192, 2, 4096, 14336, 0, 228, 220),
      (256, 2, 4096, 14336, 0, 277, 227), (250, 1, 4096, 14336, 0, 233, 212), (130, 8, 2048, 7168, 0, 118, 156),
      (224, 8, 3072, 8192, 0, 191, 205), (192, 8, 2048, 4096, 0, 98, 101), (250, 8, 2048, 4096, 0, 106, 103),
      (192, 4, 2048, 4096, 0, 88, 84), (192, 64, 2048, 1408, 0, 194, 187), (132, 60, 2048, 1408, 1, 203, 228),
      (256, 60, 2048, 1408, 1, 230, 263), (192, 8, 1024, 2816, 0, 76, 72), (192, 8, 1024, 1024, 0, 56, 44),
      (192, 128, 2048, 768, 0, 257, 200), (192, 8, 512, 1408, 0, 62, 43), (252, 32, 2048, 1408, 0, 120, 118)]


@pytest.mark.parametrize("rows,experts,d,F,shared,i8,wide", I8)
def test_integer_mma_decode_kernel_is_taken_where_it_is_the_faster_one(lib, rows, experts, d, F, shared, i8, wide):
    assert bool(lib.choice_i8_decode(rows, experts, d, F, shared)) == (i8 < wide)


def test_up_to_128_rows_the_integer_mma_decode_kernel_is_always_taken(lib):
    for rows in (1, 16, 127, 128):
        for experts, d, F in [(1, 16, 16), (8, 4096, 14336), (128, 64, 64)]:
            assert lib.choice_i8_decode(rows, experts, d, F, 0) and lib.choice_i8_decode(rows, experts, d, F, 1)


PAIRS, SINGLE, PAIR_ROWS = 0, 1, 2

# experts, rows an expert, k, us of the CTA-pair kernel, us of the single-CTA kernel
PRODUCTS = [(8, 256, 512, 27, 20), (32, 100, 512, 37, 31), (128, 16, 512, 49, 43), (128, 256, 512, 96, 66), (8, 256, 1024, 27, 25),
            (32, 256, 1024, 128, 120), (128, 100, 1024, 77, 68), (8, 64, 512, 13, 14), (8, 64, 1024, 16, 18),
            (32, 256, 1408, 69, 73), (128, 256, 1408, 216, 255), (8, 64, 2048, 18, 22), (32, 64, 2048, 74, 78),
            (32, 1024, 2048, 293, 345)]


@pytest.mark.parametrize("experts,rows,k,pair,single", PRODUCTS)
def test_pair_kernel_is_taken_where_it_is_the_faster_one(lib, experts, rows, k, pair, single):
    assert lib.choice_bf16(experts * rows, experts, k, 0) == (PAIRS if pair < single else SINGLE)


def test_large_groups_and_the_shared_expert(lib):
    for k in (16, 512, 1024):
        assert lib.choice_bf16(8 * 512, 8, k, 0) == PAIR_ROWS and lib.choice_bf16(8 * 512 - 1, 8, k, 0) == SINGLE
        assert lib.choice_bf16(1023, 1, k, 0) == PAIRS and lib.choice_bf16(1024, 1, k, 0) == PAIR_ROWS
        assert lib.choice_bf16(4095, 1, k, 1) == PAIRS and lib.choice_bf16(4096, 1, k, 1) == PAIR_ROWS
    for rows, groups in [(17, 1), (4096, 8), (1 << 30, 1), (1 << 30, 128)]:
        assert lib.choice_bf16(rows, groups, 1040, 0) == PAIRS and lib.choice_bf16(rows, groups, 1040, 1) == PAIRS


def test_the_benchmark_names_the_kernel_that_runs(lib):
    import sys
    sys.path.insert(0, ROOT)
    import bench
    from ateniaengine_b200.synth import MoeShape

    for d, F, E, k, Fs in [(512, 1408, 8, 2, 0), (1024, 512, 128, 8, 0), (2048, 1408, 60, 4, 5632), (2048, 4096, 8, 2, 0),
                           (4096, 14336, 8, 2, 0), (4096, 14336, 2, 2, 0)]:
        for rows in (1, 2, 3, 16, 17, 128, 129, 192, 240, 256, 257, 1023, 1024, 4096, 70000):
            name = bench.gate_up_kernel(MoeShape("s", d, F, E, k, True, Fs, int8=True), rows, E)
            assert (name == "grouped_gemm_decode_kernel") == (rows <= 256 and bool(lib.choice_i8_decode(rows, E, d, F, Fs > 0)))
            if name != "grouped_gemm_decode_kernel":
                assert name == ("grouped_gemm_w8_m256_kernel" if rows >= 256 * E else "grouped_gemm_w8_tmem_kernel")
            name = bench.gate_up_kernel(MoeShape("s", d, F, E, k, True, Fs), rows, E)
            if rows > 16:
                assert name == ("grouped_gemm_2cta_kernel", "grouped_gemm_tcgen05_kernel",
                                "grouped_gemm_pair_rows_kernel")[lib.choice_bf16(rows, E, d, 0)]
            else:
                assert name == ("grouped_gemv_kernel" if rows <= 2 and rows * d * F < 1 << 26 else "grouped_gemm_decode_kernel")


# rows, groups, feature tiles of the gate/up product, us of a forward with tiles of 256 / 192 / 128 / 64 token rows (0: not
# measured)
PAIR_TOKENS = [(32, 8, 112, 451, 0, 432, 422), (240, 8, 112, 464, 0, 444, 436), (512, 8, 112, 488, 0, 466, 535),
               (700, 8, 112, 519, 0, 503, 584), (64, 60, 11, 147, 0, 138, 137),
               (600, 60, 11, 209, 0, 197, 195), (1332, 60, 11, 237, 0, 223, 228), (5200, 60, 11, 309, 0, 297, 380),
               (366, 64, 11, 205, 0, 196, 196), (5400, 64, 11, 272, 0, 269, 317),
               (7800, 64, 11, 305, 302, 305, 380), (700, 8, 112, 501, 493, 490, 0), (800, 8, 112, 512, 502, 543, 0),
               (1000, 8, 112, 594, 549, 606, 0), (1200, 8, 112, 618, 674, 651, 0), (6800, 60, 11, 341, 334, 337, 0),
               (8192, 60, 11, 372, 372, 410, 0), (10000, 60, 11, 429, 442, 491, 0), (12000, 64, 11, 389, 415, 435, 0)]


@pytest.mark.parametrize("rows,groups,f_tiles,t256,t192,t128,t64", PAIR_TOKENS)
def test_pair_tile_height_is_near_the_fastest_measured(lib, rows, groups, f_tiles, t256, t192, t128, t64):
    took = {256: t256, 192: t192, 128: t128, 64: t64}[lib.choice_pair_tokens(rows, groups, f_tiles)]
    assert 0 < took <= 1.01 * min(t for t in (t256, t192, t128, t64) if t)


def test_pair_tile_height_of_one_group_holds_it_whole(lib):
    assert [lib.choice_pair_tokens(r, 1, 100) for r in (1, 64, 65, 128, 129, 4096)] == [64, 64, 128, 128, 256, 256]
    # tiles that all run at once: the lowest that do
    assert [lib.choice_pair_tokens(*a) for a in ((4096, 8, 1), (333, 1, 12), (333, 1, 13), (333, 1, 22), (333, 1, 25))] == [
        64, 64, 128, 128, 256]


# tokens, top-k, experts, d, F, shared width, us of a forward with the shared expert riding along / on its own stream
SHARED_RIDES = [(300, 1, 64, 2048, 1408, 1408, 191, 200), (600, 1, 64, 2048, 1408, 1408, 209, 222), (100, 1, 64, 2048, 1408, 5632, 152, 157),
                (300, 1, 64, 2048, 1408, 5632, 205, 203), (600, 1, 64, 2048, 1408, 5632, 237, 230), (100, 1, 64, 2048, 1408, 22528, 206, 202),
                (300, 1, 64, 2048, 1408, 22528, 276, 261), (600, 1, 64, 2048, 1408, 22528, 405, 329),
                (1000, 1, 64, 2048, 1408, 22528, 423, 405), (1480, 1, 64, 2048, 1408, 22528, 572, 530),
                (1000, 1, 64, 2048, 1408, 5632, 257, 263), (600, 2, 64, 2048, 1408, 22528, 331, 340),
                (1480, 2, 64, 2048, 1408, 22528, 591, 548), (300, 1, 128, 2048, 768, 3072, 211, 214), (1000, 1, 128, 2048, 768, 3072, 273, 261),
                (100, 1, 128, 2048, 768, 12288, 160, 165), (300, 1, 128, 2048, 768, 12288, 245, 241), (600, 1, 128, 2048, 768, 12288, 325, 287),
                (1000, 1, 128, 2048, 768, 12288, 399, 340), (600, 1, 16, 2048, 4096, 8192, 199, 215),
                (1000, 1, 16, 2048, 4096, 8192, 242, 249), (303, 1, 16, 1024, 2816, 5632, 85, 87), (500, 1, 16, 1024, 2816, 5632, 87, 93),
                (100, 2, 32, 2048, 1408, 11264, 136, 145), (600, 2, 32, 2048, 1408, 11264, 181, 193), (333, 2, 8, 512, 512, 1024, 30, 41),
                (333, 4, 60, 2048, 1408, 5632, 205, 215)]


@pytest.mark.parametrize("tokens,k,experts,d,F,Fs,along,aside", SHARED_RIDES)
def test_the_shared_expert_rides_along_where_that_is_faster(lib, tokens, k, experts, d, F, Fs, along, aside):
    tile = lib.choice_pair_tokens(tokens * k, experts, (F + 127) // 128)
    took = along if lib.choice_shared_rides(tokens, tile, d, Fs) else aside
    assert took <= 1.01 * min(along, aside)


# tokens, d, experts, us of the router kernel (or the forward where they are close) with the integer router / the f64 one
ROUTER_I8 = [(1185, 2048, 64, 21.1, 27.0), (1600, 2048, 64, 21.0, 30.5), (2368, 2048, 64, 28.1, 31.0), (4096, 2048, 64, 30.3, 54.0),
             (8192, 2048, 64, 46.6, 104), (1185, 1536, 64, 20.5, 21.3), (2368, 1536, 64, 25.3, 25.0), (2400, 1536, 64, 25.3, 42.1),
             (1600, 1536, 40, 19.4, 21.7), (2048, 1024, 64, 21.8, 19.4), (1600, 768, 64, 16.9, 14.2), (2400, 768, 64, 21.1, 24.9),
             (2048, 512, 64, 18.3, 11.7), (3000, 512, 64, 84.2, 84.2), (4096, 512, 64, 90.4, 90.4), (8192, 512, 64, 128, 138),
             (2048, 256, 64, 16.7, 8.9), (4096, 256, 64, 80, 76), (8192, 256, 64, 106.6, 109), (3000, 256, 40, 55.5, 51.4),
             (3000, 4096, 32, 40.5, 51.4), (2400, 2048, 32, 26.0, 28.0), (8192, 2048, 32, 45.4, 54.7), (4096, 1536, 32, 24.5, 23.2),
             (8192, 1536, 32, 38.3, 43.8), (4096, 1024, 32, 67.8, 65.7), (8192, 1024, 32, 102.5, 104.3), (8192, 512, 32, 77.7, 76.0),
             (4096, 256, 32, 51.4, 43.3), (2400, 2048, 20, 24.0, 27.4)]


@pytest.mark.parametrize("tokens,d,experts,i8,f64", ROUTER_I8)
def test_the_integer_router_where_it_is_faster(lib, tokens, d, experts, i8, f64):
    assert (i8 if lib.choice_router_i8(tokens, d, experts) else f64) <= 1.02 * min(i8, f64)
