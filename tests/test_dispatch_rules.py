"""The rules by which calls are sent to kernels (csrc/rules.h), compiled for the
host and checked at their limits.  CPU only."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "trove_gb300" / "csrc"

SHIM = """
#include "rules.h"
extern "C" {
int slab() { return trv::kSlab; }
unsigned most_pass_words() { return trv::kMostPassWords; }
unsigned widest_in_parts() { return trv::kWidestInParts; }
int parts(unsigned width, unsigned long long n, unsigned long long dst_n, int sectors) {
    return trv::scatter_parts(width, n, dst_n, sectors,
                              width % 4 ? trv::kPackedRows : width > 64 ? trv::kWideRows : trv::kStructRows);
}
int packed(int gather, unsigned width, unsigned long long n) { return trv::packed_form(gather, width, n); }
int rows_unroll(int gather, unsigned width, unsigned long long n) { return trv::rows_unroll(gather, width, n); }
int struct_unroll(int gather, unsigned width, unsigned long long n) { return trv::struct_unroll(gather, width, n); }
int default_unroll(unsigned width) { return trv::default_unroll(width); }
int exit_unroll(unsigned width, unsigned long long bytes) { return trv::exit_unroll(width, bytes); }
int layout_unroll(int to_soa, unsigned width, unsigned long long n) { return trv::layout_unroll(to_soa, width, n); }
unsigned least_packed() { return trv::kLeastPackedWidth; }
// tile bytes of each task (op, width, n); whether they make one wave
int tiles(const long long* tasks, long long count, int blocks, int* bytes) {
    const trv::TileRule rule([&](uint64_t k) {
        return trv::TileTask{tasks[3 * k] == 0, uint32_t(tasks[3 * k + 1]), uint64_t(tasks[3 * k + 2])};
    }, uint64_t(count), blocks);
    for (long long k = 0; k < count; ++k) bytes[k] = rule.tile_bytes(int(tasks[3 * k]), uint32_t(tasks[3 * k + 1]));
    return rule.one_wave();
}
int tuned_tile(int op, unsigned width, unsigned long long n, unsigned long long count, int tuned) {
    const trv::TileRule rule([&](uint64_t) { return trv::TileTask{op == 0, width, n}; }, count, 608);
    return rule.tile_bytes(op, width, tuned);
}
int piece_rows(int blocks_per_sm, int wide, int row_bytes) {
    return trv::piece_rows(trv::stage_bytes(blocks_per_sm), wide, row_bytes);
}
// whether the sample of idx says that the rows lie in order
int local(const int* idx, long long n, int row_bytes) {
    int near = 0;
    for (int lane = 0; lane < trv::kSamples; ++lane) {
        const long long p = trv::sample_position(lane, n);
        if (p < 0 || p + 1 >= n) return -1;
        near += trv::sample_near(idx[p], idx[p + 1], row_bytes);
    }
    return near >= trv::near_pairs(row_bytes);
}
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o",
                    str(d / "rules.so")], check=True)
    lib = ctypes.CDLL(str(d / "rules.so"))
    lib.most_pass_words.restype = ctypes.c_uint32
    lib.parts.argtypes = [ctypes.c_uint32, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int]
    lib.tiles.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    lib.tuned_tile.argtypes = [ctypes.c_int, ctypes.c_uint32, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int]
    lib.exit_unroll.argtypes = [ctypes.c_uint32, ctypes.c_uint64]
    for f in (lib.packed, lib.rows_unroll, lib.struct_unroll, lib.layout_unroll):
        f.argtypes = [ctypes.c_int, ctypes.c_uint32, ctypes.c_uint64]
    lib.local.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int]
    return lib


def test_rows_in_parts_keep_32_bit_offsets(rules):
    """A slab of the widest rows that go in parts: the words of the whole slab and
    a round past them, which the kernel counts in 32 bits with a sign."""
    most = rules.most_pass_words()
    in_flight = 32 * 8  # words that a round of a warp covers
    assert rules.slab() * most + 2 * in_flight <= 2**31 - 1
    assert rules.widest_in_parts() <= 4 * most


def test_parts_follow_the_destination_not_the_entry(rules):
    """What policy 6 comes to, whoever asked for it: nothing special on short
    destinations, on ones that are mostly not written, on more parts than pay."""
    for width in (4, 8, 12, 24, 48, 64):
        assert rules.parts(width, 1 << 14, 1 << 14, 1) == 0  # fits L2
        assert rules.parts(width, 1, 1, 1) == 0
        assert rules.parts(width, (34 << 20) // width, (34 << 20) // width, 1) == 0
    assert rules.parts(12, 1 << 24, 1 << 24, 1) == 4
    assert rules.parts(12, 1 << 24, 1 << 30, 1) == 0  # 64 parts of a destination that is mostly left alone
    assert rules.parts(24, 5 << 24, 5 << 24, 1) == 0  # 35 parts
    for width in (80, 256):
        assert rules.parts(width, 1 << 17, 1 << 17, 1) == 0  # the fetch alone does not pay for wide rows
    assert rules.parts(80, 1 << 20, 1 << 21, 1) == 0  # half of the rows written: too few to a pass
    assert rules.parts(200, 1 << 22, 1 << 22, 1) == 0
    assert rules.parts((34 << 20) + 4, 512, 3, 1) == 0
    for width in (12, 13, 24, 48):  # one pass after the fetch
        assert rules.parts(width, (41 << 20) // width, (41 << 20) // width, 0) == 1


@pytest.mark.parametrize("n", [2, 3, 31, 225, 226, 4097, 1 << 16, (1 << 16) + 32, 1 << 20, (1 << 20) - 1])
def test_sampled_order_of_indices(rules, n):
    """Rows in order, backwards, with gaps and in shuffled runs of 8 to 4096 are
    told from random ones, whatever power of two the array's length is."""
    rng = np.random.default_rng(n)

    def local(idx, row_bytes):
        idx = np.ascontiguousarray(idx, np.int32)
        return rules.local(idx.ctypes.data, len(idx), row_bytes)

    order = np.arange(n)
    for row_bytes in (12, 48, 200):
        assert local(order, row_bytes) == local(order[::-1], row_bytes) == 1
        assert local(np.sort(rng.permutation(4 * n)[:n]), row_bytes) == 1
        for run in (8, 32, 128, 4096):
            if n >= 32 * run and n % run == 0:
                runs = rng.permutation(n // run)[:, None] * run + np.arange(run)
                assert local(runs.reshape(-1), row_bytes) == 1, run
        if n >= 1 << 16:
            assert local(rng.permutation(n), row_bytes) == 0


def test_packed_words_only_where_they_are_right(rules):
    """A word has bytes of two rows at most and reads at most eight bytes past a row."""
    assert 2 * rules.least_packed() >= 8 and rules.least_packed() + 1 > 4
    for gather in (0, 1):
        for n in (1, 1 << 16, 1 << 20, 1 << 28):
            for width in (1, 2, 3, (1 << 20) + 1, 2**32 - 1):
                assert rules.packed(gather, width, n) == 0
    # long scatters of narrow rows: a thread per row where a sample finds them in order
    for width, n, scatter, gather in [(6, 1 << 12, 0, 0), (6, 1 << 18, 1, 0), (8, 1 << 20, 2, 1), (10, 1 << 20, 1, 1),
                                      (11, 1 << 16, 1, 0), (13, 16, 1, 1)]:
        assert (rules.packed(0, width, n), rules.packed(1, width, n)) == (scatter, gather), width


def test_structs_per_lane_are_built(rules):
    """Every choice is one of the unrolls built; a grid's structs per lane do not
    depend on the length."""
    for width in range(4, 65, 4):
        assert rules.default_unroll(width) in (1, 2, 4, 8)
        for n in (1, 1 << 16, (1 << 16) + 1, 1 << 22, 1 << 26):
            for gather in (0, 1):
                assert rules.rows_unroll(gather, width, n) in (1, 2, 4, 8)
                assert rules.struct_unroll(gather, width, n) in (1, 2, 4, 8)
                assert rules.layout_unroll(gather, width, n) in (1, 2, 4, 8)
            assert rules.exit_unroll(width, n * width) in (1, 2, 4, 8)
    assert [rules.default_unroll(w) for w in (8, 16, 32, 36)] == [8, 4, 2, 1]
    assert [rules.exit_unroll(16, mib << 20) for mib in (1, 16, 1024)] == [1, 4, 2]
    # fields' arrays aligned to sectors or not
    assert [rules.layout_unroll(1, 64, (1 << 23) + k) for k in (0, 1, 4, 8)] == [1, 2, 2, 1]
    assert [rules.layout_unroll(1, w, (1 << 25) + 1) for w in (32, 36, 40, 44, 48)] == [2, 1, 2, 1, 2]
    assert rules.struct_unroll(0, 8, 1 << 22) == 8 and rules.struct_unroll(1, 8, 1 << 22) == 4


def tiles_of(rules, tasks, blocks=608):
    a = np.array(tasks, np.int64).reshape(-1, 3)
    out = np.zeros(len(a), np.int32)
    one = rules.tiles(a.ctypes.data, len(a), blocks, out.ctypes.data)
    structs = np.maximum(out // a[:, 1] // 32 * 32, 32)
    return bool(one), out, -(-a[:, 2] // structs)


def test_tiles_of_a_batch(rules):
    """A batch that can be one wave of tiles is one, whatever is left over of its
    arrays; narrow rows get shorter tiles than wide ones; large batches get the largest
    tiles, and nothing gets more than that."""
    for op in (0, 1, 2):
        for width in range(4, 65, 4):
            for count, n in [(16, 1024), (16, 32768), (256, 512), (256, 2048), (100, 20000), (607, 999), (1, 1 << 18)]:
                one, size, count_of = tiles_of(rules, [(op, width, n)] * count)
                assert size.max() <= (65536 if one else (131072, 65536, 49152)[op])
                if count * n * width <= 30 << 20:
                    assert one and count_of.sum() <= 608
            assert tiles_of(rules, [(op, width, 512 if op else 8192 // width // 32 * 32)] * 256)[2].max() == 1
            one, size, _ = tiles_of(rules, [(op, width, 1 << 22)] * 40)
            assert not one and size[0] == (131072, 65536, 49152)[op]
    one, size, count_of = tiles_of(rules, [(1, 16, 8192)] * 256)  # 64 KiB and two to an array just fit
    assert one and size[0] == 65536 and count_of.sum() == 512
    _, size, _ = tiles_of(rules, [(1, 4, 30000), (1, 64, 30000)] * 20)
    assert size[0] // 4 > size[1] // 64 and size[0] < size[1]
    assert tiles_of(rules, [(1, 12, 0)] * 5)[0] and tiles_of(rules, [])[0]
    assert tiles_of(rules, [(2, 64, 32)] * 50000)[2].max() == 1


def test_staged_pieces_fit_their_memory(rules):
    for blocks in (2, 4):
        memory = 81408 if blocks == 2 else 40704
        for width in range(4, 65, 4):
            rows = rules.piece_rows(blocks, 0, width)
            assert rows % 32 == 0 and rows >= 32 and 3 * rows * width + 4 * rows * 4 <= memory
            if width % 16 == 0:
                rows = rules.piece_rows(blocks, 1, width)
                # the division of a word's number by words to a row holds for 12 bits
                assert rows % 32 == 0 and rows >= 32 and 2 * rows * (width + 4) <= memory and rows * width // 16 <= 4096


def test_tuned_tiles_do_not_outgrow_a_small_batch(rules):
    """A tuned tile is kept where the batch is large enough for the largest tiles, and
    where it is smaller than the batch's own; 0 stands for none."""
    for op in (0, 1, 2):
        for width in (4, 20, 64):
            own = rules.tuned_tile(op, width, 20000, 16, 0)
            assert own < 65536
            for tuned in (32 << 10, 64 << 10, 1 << 20):
                assert rules.tuned_tile(op, width, 20000, 16, tuned) == min(own, tuned)
                assert rules.tuned_tile(op, width, 1 << 22, 64, tuned) == tuned
