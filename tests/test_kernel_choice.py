"""Rules that choose among kernels are host arithmetic: they are compiled by the host compiler and held against measured times, so
that no call is slower than by the kernel that served all of them before. Runs without a GPU."""
import os
import subprocess

import pytest

import helpers
import two_tiles

CSRC = os.path.join(helpers.PKG_DIR, "csrc")


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    """Compiles a body of C++ lines that print one number each, and returns those."""
    def run(header, lines):
        folder = tmp_path_factory.mktemp("choice")
        src = folder / "ask.cpp"
        src.write_text('#include <cstdio>\n#include "%s"\nint main() {\n%s\n}\n' % (os.path.join(CSRC, header), "\n".join(lines)))
        exe = str(folder / "ask")
        subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe, str(src)], check=True)
        return [float(x) for x in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()]
    return run


# head size, q heads, kv heads, segments (rows, position, times), us of the tcgen05 and of the mma.sync kernel
PROMPTS = [
    (128, 32, 8, [(65, 0, 1)], 9.5, 7.6),
    (128, 32, 8, [(65, 2048, 1)], 32.9, 59.0),
    (128, 32, 8, [(256, 0, 1)], 11.8, 10.9),
    (128, 32, 8, [(512, 0, 1)], 15.9, 25.7),
    (128, 32, 8, [(65, 0, 32)], 65.1, 50.4),
    (128, 32, 8, [(65, 1024, 32)], 153.0, 324.1),
    (128, 32, 8, [(16, 0, 31), (300, 0, 1)], 72.5, 35.6),
    (128, 32, 8, [(64, 3600, 31), (300, 3600, 1)], 411.9, 598.0),
    (128, 8, 2, [(192, 0, 12)], 20.3, 13.2),
    (128, 8, 2, [(1024, 0, 4)], 37.5, 65.1),
    (64, 32, 4, [(128, 512, 1)], 13.3, 12.6),
    (64, 32, 4, [(1024, 0, 2)], 50.0, 60.4),
    (64, 32, 4, [(192, 256, 12)], 60.5, 46.2),
    (64, 32, 4, [(192, 2048, 12)], 168.5, 199.7),
    (64, 32, 4, [(64, 1024, 31), (300, 1024, 1)], 147.3, 113.3),
]


def cost(i, hd, qh, kvh, segs):
    adds = " ".join(f"c{i}.add({r}, {p}, {n});" for r, p, n in segs)
    return f"M40PromptCost c{i}({hd}, {qh}, {kvh}, 148, {max(r for r, _, _ in segs)}); {adds}"


def test_prompt_kernels_are_chosen_as_measured(ask):
    got = ask("prompt_cost.cuh", [cost(i, *p[:4]) + f' printf("%d\\n", c{i}.tc_us() < c{i}.mma_us());' for i, p in enumerate(PROMPTS)])
    for p, tc in zip(PROMPTS, got):
        assert (p[4] if tc else p[5]) <= min(1.05 * p[5], 1.25 * p[4]), p


# the same, us of the tcgen05 kernel with one and with two row tiles per CTA
ROW_TILES = [
    (128, 32, 8, [(640, 0, 1)], 18.3, 26.0),
    (128, 32, 8, [(1000, 0, 1)], 27.3, 35.4),
    (128, 32, 8, [(1300, 0, 1)], 44.8, 43.2),
    (128, 32, 8, [(2048, 0, 1)], 76.0, 68.3),
    (128, 32, 8, [(640, 1000, 1)], 42.3, 52.2),
    (128, 32, 8, [(1000, 4000, 1)], 121.8, 137.4),
    (128, 32, 8, [(500, 0, 4)], 44.7, 36.6),
    (128, 32, 8, [(700, 0, 3)], 52.4, 44.5),
    (128, 16, 2, [(1300, 0, 1)], 23.5, 41.8),
    (128, 16, 2, [(2048, 0, 1)], 37.3, 60.7),
    (128, 16, 2, [(1024, 0, 4)], 54.4, 46.3),
    (128, 16, 2, [(1500, 0, 1), (200, 0, 1), (300, 0, 1)], 32.8, 46.6),
    (64, 32, 4, [(1000, 0, 1)], 22.0, 27.8),
    (64, 32, 4, [(2048, 0, 1)], 60.7, 53.0),
    (64, 32, 4, [(1000, 4000, 1)], 104.0, 112.2),
    (64, 32, 4, [(500, 0, 4)], 34.0, 26.3),
    (64, 40, 40, [(820, 0, 1)], 21.8, 25.9),
    (64, 40, 40, [(1500, 0, 1)], 49.5, 46.4),
    (64, 40, 40, [(1000, 4000, 1)], 154.7, 191.7),
    (64, 40, 40, [(65, 2000, 16)], 140.0, 250.3),
    (64, 40, 40, [(1024, 0, 4)], 105.1, 97.5),
    (128, 33, 11, [(2048, 0, 1)], 78.4, 77.6),
    (128, 33, 11, [(65, 2000, 16)], 132.4, 239.2),
    (128, 33, 11, [(1000, 0, 1)], 28.2, 37.7),
    (128, 8, 2, [(1024, 0, 4)], 27.4, 35.8),
]


def test_row_tiles_per_cta_are_chosen_as_measured(ask):
    got = ask("prompt_cost.cuh", [cost(i, *p[:4]) + f' printf("%d\\n", c{i}.tc_two());' for i, p in enumerate(ROW_TILES)])
    for p, two in zip(ROW_TILES, got):
        assert (p[5] if two else p[4]) <= 1.05 * min(p[4:]), p
    assert sum(got) >= 8


def test_calls_that_test_two_row_tiles_have_them(ask):
    cases = [(hd, qh, kvh, [(q, kv - q, 1) for q, kv in pairs]) for qh, kvh, hd, pairs in two_tiles.PACKED]
    cases += [(hd, qh, kvh, [(rows, pos, 1)]) for qh, kvh, hd, pos, rows in two_tiles.CACHED]
    cases += [(64 if max(d, v) <= 64 else 128, h, g, [(rows, 0, 1)]) for h, g, d, v, rows in two_tiles.STACKS]
    assert all(ask("prompt_cost.cuh", [cost(i, *p) + f' printf("%d\\n", c{i}.tc_two() && c{i}.tc_us() < c{i}.mma_us());' for i, p in enumerate(cases)]))


# the same, us of the faster prompt kernel and of the decode form (a row reads its own context)
PORTIONS = [
    (128, 32, 8, [(16, 0, 1)], 5.7, 10.2),
    (128, 32, 8, [(16, 1024, 1)], 31.3, 24.5),
    (128, 32, 8, [(16, 8192, 1)], 209.9, 70.6),
    (128, 32, 8, [(32, 2048, 2)], 56.8, 80.8),
    (128, 32, 8, [(64, 8192, 1)], 210.0, 239.3),
    (128, 32, 8, [(256, 8192, 1)], 106.0, 940.7),
    (128, 16, 2, [(48, 4096, 1)], 107.8, 38.8),
    (128, 16, 2, [(65, 8192, 1)], 102.0, 75.3),
    (128, 16, 2, [(16, 2048, 12)], 88.0, 69.5),
    (128, 16, 2, [(256, 2048, 2)], 34.7, 168.4),
    (64, 32, 4, [(16, 8192, 1)], 113.6, 26.3),
    (64, 32, 4, [(64, 4096, 1)], 58.9, 45.6),
    (64, 32, 4, [(32, 512, 4)], 11.3, 29.7),
    (64, 32, 4, [(128, 4096, 4)], 45.5, 288.3),
    (64, 8, 8, [(24, 8192, 2)], 112.7, 93.7),
    (64, 8, 8, [(24, 1024, 12)], 18.4, 100.8),
]


def test_portions_of_prompts_take_the_form_that_was_faster(ask):
    got = ask("prompt_cost.cuh", [cost(i, *p[:4]) + f' printf("%d\\n", c{i}.prompt_us() < c{i}.decode_us());' for i, p in enumerate(PORTIONS)])
    for p, prompt in zip(PORTIONS, got):
        assert (p[4] if prompt else p[5]) <= 1.05 * p[5], p
    assert sum(got) >= 7  # and those that gain much do take the prompt form


# rows, outputs of gate and of up, K: us of shared tiles, of two problems with K splits
GATE_UP = [(200, 640, 8192, 73.1, 25.0), (160, 4096, 2048, 28.4, 22.0), (129, 64, 2048, 23.0, 12.3), (512, 1408, 2048, 28.4, 23.7), (300, 2048, 8192, 86.8, 51.4),
           (256, 8192, 64, 13.8, 27.3), (129, 8192, 256, 12.4, 21.2), (2048, 8192, 64, 59.3, 139.6), (1030, 4096, 2048, 81.9, 86.2)]


def test_gate_up_calls_are_cut_as_measured(ask):
    got = ask("gemm_tc_pair_plan.cuh", ["M40PairPlan p;"] + [
        f'{{ const int n[2] = {{{n}, {n}}}; m40_pair_cut_best(74, {m}, {(k + 63) // 64}, 2, n, true, false, &p); printf("%d\\n", p.paired); }}'
        for m, n, k, _, _ in GATE_UP])
    for case, shared in zip(GATE_UP, got):
        assert (case[3] if shared else case[4]) == min(case[3:]), case


# head size, heads, segments, tokens of each; us of the call a token at a time in CTAs of 32 columns, then of the scan in pairs with 16 lanes
# and 2 columns, 8 and 2, 8 and 4, each with one, two and three CTAs per SM at most
SCANS = [
    (64, 32, 1, 2048, 368.3, [[301.1, 382.6, 493.1], [330.1, 493.3, 692.4], [475.5, 758.7, 980.5]]),
    (64, 16, 3, 200, 42.0, [[61.2, 44.5, 55.4], [39.2, 55.1, 74.7], [53.4, 81.0, 84.4]]),
    (64, 16, 6, 100, 43.4, [[50.9, 45.6, 34.4], [40.8, 34.0, 44.0], [33.0, 46.9, 62.6]]),
    (64, 32, 2, 300, 63.4, [[92.0, 67.5, 83.9], [59.6, 83.5, 112.7], [81.1, 122.0, 168.9]]),
    (64, 32, 4, 300, 126.9, [[182.4, 132.3, 134.3], [117.8, 99.7, 128.9], [97.2, 138.3, 185.2]]),
    (64, 64, 1, 256, 54.2, [[78.7, 57.7, 71.8], [51.1, 71.5, 96.6], [69.2, 104.6, 113.0]]),
    (64, 64, 16, 94, 300.1, [[432.9, 306.3, 275.1], [281.9, 227.6, 218.6], [229.7, 193.1, 187.1]]),
    (64, 75, 1, 300, 113.1, [[131.3, 105.6, 86.4], [103.6, 86.2, 115.5], [83.7, 125.0, 171.7]]),
    (64, 48, 12, 50, 96.2, [[143.3, 101.3, 91.5], [92.5, 74.4, 71.5], [74.1, 63.2, 61.6]]),
    (64, 32, 1, 33, 11.6, [[12.1, 12.6, 14.5], [11.4, 14.3, 17.8], [13.7, 18.5, 18.4]]),
    (32, 32, 12, 50, 32.0, [None, [31.5, 31.5, 25.7], [33.5, 33.5, 30.5]]),
    (32, 64, 32, 33, 86.7, [None, [86.9, 86.9, 81.3], [98.4, 98.4, 90.2]]),
    (96, 24, 3, 200, 101.9, [None, [90.0, 79.6, 108.1], [72.3, 108.4, 146.1]]),
    (96, 24, 24, 33, 123.8, [None, [116.5, 94.0, 90.7], [110.9, 89.8, 85.7]]),
    (128, 16, 1, 300, 105.6, [[55.1, 80.8], [76.0, 125.4], [114.2, 188.4]]),
    (128, 36, 1, 300, 110.4, [[104.8, 87.4], [82.8, 132.7], [121.8, 181.5]]),
    (128, 64, 1, 300, 216.6, [[207.6, 171.5], [164.4, 150.2], [139.2, 213.3]]),
    (128, 16, 16, 100, 267.3, [[263.9, 207.7], [206.4, 179.9], [189.8, 162.8]]),
    (160, 8, 1, 300, 146.1, [[64.7], [112.8], None]),
    (160, 30, 1, 300, 290.5, [[184.5], [225.5], None]),
    (192, 16, 2, 300, 297.4, [[194.6], [235.2], None]),
    (192, 16, 24, 33, 303.0, [[288.0], [258.5], None]),
    (256, 9, 1, 300, 301.7, [[81.9], [146.1], None]),
    (256, 19, 1, 300, 589.4, [[221.1], [287.0], None]),
    (256, 16, 24, 33, 759.9, [[442.3], [418.5], None]),
]


def test_delta_scans_take_the_form_that_was_fastest(ask):
    got = ask("delta_scan_plan.cuh", [f'{{ const M40ScanPlan p = m40_scan_plan({d}, {h}, {s}, {s * n}, {n}, 148); printf("%u %u %u\\n", p.lanes, p.cols, p.per_sm); }}'
                                      for d, h, s, n, _, _ in SCANS])
    for case, (lanes, cols, per) in zip(SCANS, zip(*[iter(got)] * 3)):
        times = case[5][{(16, 2): 0, (8, 2): 1, (8, 4): 2}[lanes, cols]]
        assert times[int(per) - 1] <= 1.06 * min(t for f in case[5] if f for t in f), case
        assert times[int(per) - 1] <= case[4], case


def test_single_tokens_beside_a_prompt_do_not_choose_its_scan(ask):
    """A step of 31 decoding sequences and one prompt: the prompt's chain is what takes long."""
    alone, beside = ask("delta_scan_plan.cuh", [f'{{ const M40ScanPlan p = m40_scan_plan(64, 32, {s}, {r}, 300, 148); printf("%u\\n", p.lanes * 100 + p.cols); }}'
                                                for s, r in ((1, 300), (32, 331))])
    assert alone == 1602 and beside == 802
