"""Rules that choose between kernels, on the host: no GPU is needed to ask them."""
import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "vlrf_b200" / "csrc"


@pytest.mark.parametrize("H,lens,parts,listed", [
    # whole prompt steps measured: listed tiles were faster here …
    (25, [1013, 517, 389, 97, 31, 1, 1, 1], 1, True), (20, [3, 28, 4, 124, 12, 466, 1, 1, 1, 1, 1], 1, True), (25, [469, 154, 12, 1, 1, 1, 1, 1], 1, True),
    # … and slower here: the tiles leave SMs idle, or hardly any place is saved
    (12, [92, 32, 102, 632, 40, 10, 1, 1, 1, 1, 1], 1, False), (12, [900, 200, 77, 10, 1, 1, 1, 1, 1], 1, False), (25, [344, 4, 538], 1, False),
    (16, [3, 36, 49, 122, 576, 40, 1, 1, 1, 1, 1], 1, False), (20, [16, 627, 857, 1], 1, False), (16, [600, 500, 400, 300], 1, False),
    (64, [2000], 1, False), (64, [1000] + [1] * 32, 1, False), (64, [8193] + [1] * 20, 1, False)])
def test_prompt_tiles_are_listed_only_where_they_fill_the_gpu(H, lens, parts, listed):
    from vlrf_b200.csrc import library
    assert bool(library().vlrf_attn_prefill_tc_lists(sum(lens), len(lens), max(lens), H, parts, 148)) == listed


@pytest.mark.parametrize("rows,G,N,width", [
    (2000, 16, 1024, 128), (1000, 16, 2048, 128), (4096, 16, 1024, 128), (4096, 16, 2048, 256), (5000, 8, 64, 64), (5000, 8, 128, 128)])
def test_wide_tiles_of_experts_only_where_full_tiles_gain_too(rows, G, N, width):
    """2,000 rows over 16 experts are 16 full row tiles of 128, one round of narrow tiles; counted with a half-empty tile a group they
    looked like two."""
    from vlrf_b200.csrc import library
    assert library().vlrf_gemm_tcgen05_groups_width(rows, G, N, 1, 148) == width


@pytest.mark.parametrize("M,N,rows", [
    (2048, 768, 96), (2048, 2304, 256), (2048, 3072, 192), (2050, 1600, 224), (2050, 4800, 192), (2050, 6400, 192), (1928, 11264, 256),
    (1500, 1280, 128), (700, 3072, 128), (512, 768, 64), (65, 256, 64)])
def test_rows_of_a_tile_of_a_pair(M, N, rows):
    """The rows with which each of these was fastest (or within 5 %)."""
    from vlrf_b200.csrc import library
    assert library().vlrf_gemm_pair_rows(M, N, 148) == rows


def test_rows_of_a_tile_of_a_pair_cost_the_same_to_find_on_any_gpu():
    """Every many-row product asks.  The pair that has most to do is always the first, so nothing is gone through pair by pair: the same rows as where it
    is, and no more time for 268 million pairs than for 74."""
    import random
    import time
    from vlrf_b200.csrc import library

    def by_pair(M, N, sms):
        pairs, tiles_w, best = max(1, sms // 2), -(-N // 256), None
        for bn in range(256, 63, -32):
            whole, left = M // bn * tiles_w, (M % bn + 31) // 32 * 32
            tiles = whole + (tiles_w if left else 0)
            most = 0
            for p in range(pairs):
                mine, of_all = whole // pairs + (p < whole % pairs), tiles // pairs + (p < tiles % pairs)
                most = max(most, mine * (bn + 96) + (of_all - mine) * (left + 96))
            if best is None or most < best[0]:
                best = (most, bn)
        return best[1]

    r = random.Random(5)
    for _ in range(3000):
        M, N, sms = int(2 ** r.uniform(6, 15)), int(2 ** r.uniform(3, 16)), r.choice([148, 148, 132, 8, 3, 1])
        assert library().vlrf_gemm_pair_rows(M, N, sms) == by_pair(M, N, sms), (M, N, sms)
    t0 = time.perf_counter()
    library().vlrf_gemm_pair_rows(2048, 2304, 2 ** 29)
    assert time.perf_counter() - t0 < 0.1


@pytest.mark.parametrize("M,N,K,dtype,rows", [
    # measured faster by pairs of SMs …
    (2048, 768, 768, 0, 96), (2048, 768, 3072, 0, 96), (512, 768, 768, 0, 64), (2050, 1600, 1600, 0, 224), (2050, 1600, 6400, 0, 224), (4096, 4096, 4096, 0, 256),
    (1024, 11264, 2048, 0, 224), (65, 16, 1024, 0, 64), (128, 6144, 2048, 0, 64), (1928, 11264, 2048, 1, 256), (4096, 4096, 4096, 1, 256), (512, 4096, 4096, 1, 128), (777, 8192, 3072, 1, 224),
    (512, 8192, 3072, 1, 256), (2050, 11264, 2048, 1, 256), (777, 2048, 4096, 1, 96),
    # … and by one CTA a tile: little work for 2-byte columns, tiles of 160 to 224 rows along a long K, rows that fill no tile of 192
    (2048, 2304, 768, 1, 0), (512, 4096, 1024, 1, 0), (1928, 4096, 1024, 1, 0), (2048, 3072, 1024, 1, 0), (2050, 4800, 1600, 1, 0), (1024, 6144, 2048, 1, 0), (2048, 1600, 6400, 1, 0), (3000, 2048, 2048, 1, 0),
    (128, 11264, 2048, 1, 0), (240, 11264, 2048, 1, 0), (240, 11264, 2048, 0, 0), (2048, 1280, 5120, 0, 0), (1500, 1600, 6400, 0, 0), (2048, 1600, 6400, 0, 0)])
def test_products_by_pairs_only_where_they_gain(M, N, K, dtype, rows):
    """Float32 (0) and bfloat16 (1) results; the rows of a pair's tile, 0 for one CTA a tile."""
    from vlrf_b200.csrc import library, ops
    assert (ops.F32, ops.BF16) == (0, 1)
    assert library().vlrf_gemm_tcgen05_pair_rows(M, N, K, dtype, 148) == rows


@pytest.mark.parametrize("M,N,K,gains", [
    # measured faster with the norm ahead: GPT-2 small up to 8 rows, medium up to 4 (and 1 row of its feed-forward) …
    (1, 2304, 768, True), (4, 3072, 768, True), (8, 2304, 768, True), (8, 3072, 768, True), (1, 3072, 1024, True), (4, 3072, 1024, True), (1, 4096, 1024, True),
    # … and slower, or no faster, where a second round of CTAs is needed; nine rows and 1,280 columns are not taken
    (5, 3072, 1024, False), (8, 3072, 1024, False), (2, 4096, 1024, False), (4, 4096, 1024, False), (8, 4096, 1024, False), (9, 768, 768, False), (1, 3840, 1280, False)])
def test_float32_norm_ahead_of_a_product_only_where_its_ctas_find_room(M, N, K, gains):
    from vlrf_b200.csrc import library
    assert bool(library().vlrf_gemm_f32_norm_gains(M, N, K, 148)) == gains


@pytest.mark.parametrize("M,N,K,then,exchanged", [
    # alone: wide products from four rows on, a vocabulary always
    (4, 7296, 1024, "kernels", True), (3, 7296, 1024, "kernels", False), (8, 8192, 2048, "kernels", False), (1, 50257, 768, "product", True),
    # the next product reads the result: measured slower up to 16 rows
    (4, 11264, 2048, "product", False), (16, 12288, 2048, "product", False), (24, 12288, 2048, "product", True), (64, 5632, 1024, "product", True),
    # a gate and the next product read it
    (4, 4224, 768, "gate", False), (8, 7040, 1280, "gate", False), (9, 9600, 1600, "gate", False), (8, 11264, 2048, "gate", True),
    (12, 5632, 1024, "gate", True), (14, 12288, 1024, "gate", False), (10, 14336, 2048, "gate", False), (16, 11264, 2048, "gate", True),
    (17, 14336, 2048, "gate", True)])
def test_wide_products_of_few_rows_by_what_reads_them(M, N, K, then, exchanged):
    from vlrf_b200.csrc import ops
    assert ops._swapped_takes(M, N, K, then) == exchanged


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_a_kernel_is_prepared_once_on_every_device(tmp_path):
    """Shared memory beyond 48 KB is granted per device: the second device of a process asks too, a failed grant is asked for again, and
    the kernels of the float32 product and of the chunked recurrence ask this way."""
    (tmp_path / "t.cpp").write_text('''
#include "device_marks.h"
#include <cassert>
int main() {
    static DeviceMarks marks, other;
    int asked[70] = {0}, answer = 0;
    auto ask = [&](DeviceMarks& m, int device) { return m.once(device, [&] { ++asked[device]; return answer; }); };
    assert(ask(marks, 0) == 0 && ask(marks, 0) == 0 && asked[0] == 1);
    assert(ask(marks, 1) == 0 && asked[1] == 1 && ask(marks, 0) == 0 && ask(marks, 1) == 0 && asked[0] == 1 && asked[1] == 1);
    answer = 7;
    assert(ask(marks, 63) == 7 && ask(marks, 63) == 7 && asked[63] == 2);
    answer = 0;
    assert(ask(marks, 63) == 0 && ask(marks, 63) == 0 && asked[63] == 3);
    assert(ask(marks, 64) == 0 && ask(marks, 64) == 0 && asked[64] == 2);
    assert(ask(other, 0) == 0 && asked[0] == 2);
    return 0;
}
''')
    subprocess.run(["g++", "-std=c++17", "-I", str(SRC), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True)
    for name in ("gemm_simt.cu", "state_chunks.cu"):
        text = (SRC / name).read_text()
        assert "static bool" not in text and "cudaFuncSetAttribute" not in text and "allow_shared_memory(" in text


@pytest.mark.parametrize("name", ["attention_prefill_tc.cu", "gemm_pair.cu", "gemm_splitk.cu", "gemm_tcgen05.cu"])
def test_warps_that_go_on_together_wait_with_one_answer(name):
    """`elect.sync`, `tcgen05.ld` and shuffles want all 32 lanes of a warp, so a wait ahead of them gives one answer to all of them; a wait of a lane's
    own, and a look at the flag that calls a CTA's work off, stand only where one lane acts."""
    import re
    text = re.sub(r"//[^\n]*", "", (SRC / name).read_text())
    scopes, statement = [], ""                       # the text ahead of each open brace; the text since the last brace or semicolon
    for piece in re.split(r"([{};])", text):
        if piece == "{":
            scopes.append(statement)
            statement = ""
        elif piece == "}":
            scopes.pop()
            statement = ""
        elif piece == ";":
            statement = ""
        else:
            statement += piece
            if re.search(r"tbar_wait_or_abort\(|\*\(volatile int\*\)&?s_abort", statement):
                alone = any(re.search(r"elect_one\(\)|\b(lane|threadIdx\.x) == 0", s) for s in scopes + [statement])
                assert alone, f"{name}: {' '.join(statement.split())}"
    assert not scopes and "tbar_wait_warp(" in text


@pytest.mark.parametrize("name", ["attention_prefill_tc.cu", "gemm_pair.cu"])
def test_kernels_that_give_up_wait_for_what_is_under_way(name):
    """Whichever role gave up: behind the place where all roles meet, and ahead of giving tensor memory back; nowhere inside a role."""
    import re
    text = re.sub(r"//[^\n]*", "", (SRC / name).read_text())
    calls = [m.start() for m in re.finditer(r"if \(\*?s_abort\)\s+\w+_drain\(", text)]
    given_back = [m.start() for m in re.finditer(r"tcgen05\.dealloc", text)]
    assert len(calls) == len(given_back) == 1 and calls[0] < given_back[0]
    assert re.search(r"(__syncthreads|cluster_sync_all)\(\);[^{}]*$", text[:calls[0]])
