"""GPU parity: every C ABI path against the CPU oracle, bit-exact, through
the C ABI.  Sizes are small enough for the oracle to finish in seconds; the
full-size workloads are checked through size-independent properties in
test_gpu_fullsize.py."""
import ctypes

import numpy as np
import pytest

import oracle
import trove_gb300 as tg

pytestmark = pytest.mark.gpu

WIDTHS = list(range(4, 65, 4))
SENTINEL = 0xA5


def to_dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()


def to_host(t):
    return t.cpu().numpy()


def guarded(torch, nbytes, offset=0, guard=256):
    """Device byte buffer with sentinel guard bands; returns (buffer, view
    start) so writes outside [start, start + nbytes) can be detected."""
    buf = torch.full((guard + offset + nbytes + guard,), SENTINEL, dtype=torch.uint8, device="cuda")
    return buf, guard + offset


def check_guards(buf, start, nbytes):
    h = to_host(buf)
    assert (h[:start] == SENTINEL).all(), "write before the destination"
    assert (h[start + nbytes:] == SENTINEL).all(), "write past the destination"
    return h[start:start + nbytes]


class KernelNodeParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def launched_grids(torch, run):
    """Blocks of each kernel that run() launches, read from a captured graph."""
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        run()
    cu, graph = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(g.raw_cuda_graph())
    count = ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    grids = []
    for node in nodes:
        kind, p = ctypes.c_int(-1), KernelNodeParams()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:  # a kernel
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            grids.append(p.grid[0])
    return grids


@pytest.mark.parametrize("width", WIDTHS)
def test_copy_struct_paths(cuda, width):
    torch = cuda
    for n in [1, 31, 33, 4097, 65539]:
        src_h = oracle.random_structs(n, width, seed=width * 1000 + n)
        src = to_dev(torch, src_h)
        expect = oracle.copy(src_h, n, width)
        for path in ["warp", "block", "direct", "vector", "auto", "bulk"]:
            for unroll in ([1, 2, 4, 8] if path in ("warp", "block", "direct", "vector") else [0]):
                for chunk in ([0, 4096, 48 << 10] if path == "bulk" else [0]):
                    buf, start = guarded(torch, n * width)
                    tg.copy(buf[start:], src, n, width, path=path, unroll=unroll, chunk=chunk)
                    got = check_guards(buf, start, n * width)
                    assert np.array_equal(got, expect), (width, n, path, unroll, chunk)
    tg.check_device()


@pytest.mark.parametrize("offset", [4, 8, 12])
@pytest.mark.parametrize("width", [8, 12, 16, 24, 32, 48, 64])
def test_copy_misaligned(cuda, width, offset):
    """Struct arrays not aligned to their widest word; the flat path with
    source and destination at different alignments."""
    torch = cuda
    n = 3001
    src_h = oracle.random_structs(n, width, seed=offset * 7 + width)
    sbuf, sstart = guarded(torch, n * width, offset=offset)
    sbuf[sstart:sstart + n * width] = to_dev(torch, src_h)
    for path in ["warp", "block", "vector", "auto", "bulk"]:
        for doff in [(offset * 3) % 16, offset]:
            dbuf, dstart = guarded(torch, n * width, offset=doff)
            if path == "bulk" and doff % 16 != offset % 16:
                with pytest.raises(tg.TroveError, match="alignment"):
                    tg.copy(dbuf[dstart:], sbuf[sstart:], n, width, path=path)
                continue
            tg.copy(dbuf[dstart:], sbuf[sstart:], n, width, path=path)
            got = check_guards(dbuf, dstart, n * width)
            assert np.array_equal(got, src_h.reshape(-1)), (path, width, offset, doff)
    tg.check_device()


@pytest.mark.parametrize("nbytes_width", [(1, 1), (3, 7), (5, 3), (100, 13), (7, 132), (1000, 100)])
def test_copy_odd_widths(cuda, nbytes_width):
    torch = cuda
    n, width = nbytes_width
    src_h = np.frombuffer(oracle.random_words((n * width + 3) // 4, 9).tobytes()[:n * width], np.uint8)
    src = to_dev(torch, src_h)
    buf, start = guarded(torch, n * width, offset=1)
    tg.copy(buf[start:], src, n, width)
    assert np.array_equal(check_guards(buf, start, n * width), src_h)
    with pytest.raises(tg.TroveError):
        tg.copy(buf[start:], src, n, width, path="warp")


@pytest.mark.parametrize("path", ["warp", "block"])
@pytest.mark.parametrize("width", WIDTHS)
def test_copy_exit(cuda, width, path):
    torch = cuda
    for n, modulus in [(20000, 7), (100003, 625), (4096, 0), (77, 3)]:
        src_h = oracle.random_structs(n, width, seed=width + n + modulus)
        init = np.full(n * width, SENTINEL, np.uint8)
        expect, written = oracle.copy_exit(init, src_h, n, width, modulus)
        src = to_dev(torch, src_h)
        dst = to_dev(torch, init)
        tg.copy_exit(dst, src, n, width, modulus, path=path)
        assert np.array_equal(to_host(dst), expect), (width, n, modulus, path)
        if modulus == 625:
            assert 0 < n - written < n // 100


def index_sets(n, seed):
    return {
        "perm": oracle.permutation(n, seed),
        "runs": oracle.run_indices(n, seed),
        "uniform": oracle.uniform_indices(n, n, seed),
        "identity": np.arange(n, dtype=np.int32),
    }


@pytest.mark.parametrize("width", WIDTHS)
def test_gather(cuda, width):
    torch = cuda
    for n in [33, 5000, 65536 + 17]:
        src_h = oracle.random_structs(n, width, seed=width * 31 + n)
        src = to_dev(torch, src_h)
        init = np.full(n * width, SENTINEL, np.uint8)
        for name, idx_h in index_sets(n, seed=n + width).items():
            idx = torch.from_numpy(idx_h).cuda()
            expect = oracle.gather(init, src_h, idx_h, n, width)
            for path in ["warp", "coalesced", "direct", "auto", "vector"]:
                for unroll in ([1, 2, 4, 8] if path in ("warp", "coalesced", "direct") else [0]):
                    dst = to_dev(torch, init)
                    tg.gather(dst, src, n, idx, n, width, path=path, unroll=unroll)
                    assert np.array_equal(to_host(dst), expect), (width, n, name, path, unroll)


@pytest.mark.parametrize("width", [4, 8, 12, 24, 64, 100])
def test_row_form_cache_policies(cuda, width):
    """Every cache policy of the row-form gather / scatter moves the same
    bytes as the oracle."""
    torch = cuda
    n = 65536 + 17
    src_h = oracle.random_structs(n, width, seed=width + 3)
    src = to_dev(torch, src_h)
    init = np.full(n * width, SENTINEL, np.uint8)
    sets = index_sets(n, seed=width)
    for policy in range(6):
        for name, idx_h in sets.items():
            idx = torch.from_numpy(idx_h).cuda()
            dst = to_dev(torch, init)
            tg.gather(dst, src, n, idx, n, width, path="warp", policy=policy)
            assert np.array_equal(to_host(dst), oracle.gather(init, src_h, idx_h, n, width)), (policy, name)
    perm_h = sets["perm"]
    for policy in range(7):
        dst = to_dev(torch, init)
        tg.scatter(dst, n, src, torch.from_numpy(perm_h).cuda(), n, width, path="warp", policy=policy)
        assert np.array_equal(to_host(dst), oracle.scatter(init, src_h, perm_h, n, width)), policy
    with pytest.raises(tg.TroveError):
        tg.gather(dst, src, n, idx, n, width, path="warp", policy=6)
    with pytest.raises(tg.TroveError):
        tg.scatter(dst, n, src, torch.from_numpy(perm_h).cuda(), n, width, path="warp", policy=7)


@pytest.mark.parametrize("width", [8, 12, 20, 24])
def test_scatter_destination_passes(cuda, width):
    """Scatters onto destinations above 64 MiB in destination passes (cache
    policy 6; the default for structs of at most 16 bytes): every row lands
    once, skipped indices leave the destination alone, a partial scatter
    keeps the rest."""
    torch = cuda
    n = (1 << 23) + 17  # 8-24 B: 64-192 MiB destinations, 2-3 passes
    src_h = oracle.random_structs(n, width, seed=width + 40)
    src = to_dev(torch, src_h)
    idx_h = oracle.permutation(n, width + 41)
    idx_h[5] = -1
    idx_h[77] = n + 3
    ok = (idx_h >= 0) & (idx_h < n)
    expect = np.full((n, width), SENTINEL, np.uint8)
    expect[idx_h[ok]] = src_h[ok]
    idx = torch.from_numpy(idx_h).cuda()
    for kw in ({}, {"path": "warp", "policy": 6}, {"path": "warp", "policy": 1}):
        dst = torch.full((n * width,), SENTINEL, dtype=torch.uint8, device="cuda")
        tg.scatter(dst, n, src, idx, n, width, **kw)
        assert np.array_equal(to_host(dst).reshape(n, width), expect), kw
    # a third of the rows, in passes on request
    m = n // 3
    expect = np.full((n, width), SENTINEL, np.uint8)
    sel = idx_h[:m]
    okm = (sel >= 0) & (sel < n)
    expect[sel[okm]] = src_h[:m][okm]
    dst = torch.full((n * width,), SENTINEL, dtype=torch.uint8, device="cuda")
    tg.scatter(dst, n, src, idx, m, width, path="warp", policy=6)
    assert np.array_equal(to_host(dst).reshape(n, width), expect)


@pytest.mark.parametrize("width", [4, 12, 16, 36, 64])
def test_gather_out_of_range_indices_are_skipped(cuda, width):
    torch = cuda
    n = 4099
    src_h = oracle.random_structs(n, width, seed=5)
    idx_h = oracle.uniform_indices(n, n, 6)
    bad = np.arange(n) % 97 == 3
    idx_h = idx_h.copy()
    idx_h[bad] = np.where(np.arange(bad.sum()) % 2 == 0, -5, n + 10)
    init = np.full(n * width, SENTINEL, np.uint8)
    expect = init.reshape(n, width).copy()
    expect[~bad] = src_h[idx_h[~bad]]
    for path in ["warp", "coalesced", "direct", "vector"]:
        dst = to_dev(torch, init)
        tg.gather(dst, to_dev(torch, src_h), n, torch.from_numpy(idx_h).cuda(), n, width, path=path)
        assert np.array_equal(to_host(dst), expect.reshape(-1)), path


@pytest.mark.parametrize("width", WIDTHS)
def test_scatter(cuda, width):
    torch = cuda
    for n in [33, 5000, 65536 + 17]:
        src_h = oracle.random_structs(n, width, seed=width * 17 + n)
        src = to_dev(torch, src_h)
        init = np.full(n * width, SENTINEL, np.uint8)
        for name in ["perm", "identity"]:
            idx_h = index_sets(n, seed=n)[name]
            idx = torch.from_numpy(idx_h).cuda()
            expect = oracle.scatter(init, src_h, idx_h, n, width)
            for path in ["warp", "coalesced", "direct", "auto", "vector"]:
                for unroll in ([1, 2, 4, 8] if path in ("warp", "coalesced") else [0]):
                    dst = to_dev(torch, init)
                    tg.scatter(dst, n, src, idx, n, width, path=path, unroll=unroll)
                    assert np.array_equal(to_host(dst), expect), (width, n, name, path, unroll)


def test_scatter_out_of_range_indices_are_skipped(cuda):
    torch = cuda
    n, width = 2000, 20
    src_h = oracle.random_structs(n, width, seed=8)
    idx_h = oracle.permutation(n, 9).copy()
    idx_h[::13] = -1
    keep = idx_h >= 0
    init = np.full(n * width, SENTINEL, np.uint8)
    expect = init.reshape(n, width).copy()
    expect[idx_h[keep]] = src_h[keep]
    for path in ["warp", "coalesced", "direct", "vector"]:
        dst = to_dev(torch, init)
        tg.scatter(dst, n, to_dev(torch, src_h), torch.from_numpy(idx_h).cuda(), n, width, path=path)
        assert np.array_equal(to_host(dst), expect.reshape(-1)), path


@pytest.mark.parametrize("width", [8, 12, 16, 24, 32, 48, 64])
def test_index_ops_misaligned(cuda, width):
    """Source and destination 4 bytes past a 16-byte boundary: the row-form
    kernels drop to 4-byte words, the coalesced_ptr kernels to the widest
    word every pointer allows."""
    torch = cuda
    n = 3001
    src_h = oracle.random_structs(n, width, seed=width)
    sbuf = torch.zeros(n * width + 64, dtype=torch.uint8, device="cuda")
    sbuf[4:4 + n * width] = to_dev(torch, src_h)
    idx_h = oracle.permutation(n, 3)
    idx = torch.from_numpy(idx_h).cuda()
    init = np.full(n * width, SENTINEL, np.uint8)
    g_expect = oracle.gather(init, src_h, idx_h, n, width)
    s_expect = oracle.scatter(init, src_h, idx_h, n, width)
    for path in ["warp", "coalesced", "direct", "auto"]:
        dbuf = torch.full((n * width + 64,), SENTINEL, dtype=torch.uint8, device="cuda")
        tg.gather(dbuf[4:], sbuf[4:], n, idx, n, width, path=path)
        assert np.array_equal(to_host(dbuf)[4:4 + n * width], g_expect), ("gather", path)
        dbuf.fill_(SENTINEL)
        tg.scatter(dbuf[4:], n, sbuf[4:], idx, n, width, path=path)
        assert np.array_equal(to_host(dbuf)[4:4 + n * width], s_expect), ("scatter", path)


def test_fill_matches_oracle_stream(cuda):
    torch = cuda
    for nwords, seed in [(1, 0), (1000, 0), (1 << 20, 12345)]:
        t = torch.empty(nwords, dtype=torch.int32, device="cuda")
        tg.fill_random_u32(t, nwords, seed)
        assert np.array_equal(to_host(t).view(np.uint32), oracle.random_words(nwords, seed))


def test_uniform_indices_match_oracle(cuda):
    torch = cuda
    for n, bound, seed in [(1, 1, 0), (5000, 77, 3), (1 << 20, 1 << 20, 9)]:
        t = torch.empty(n, dtype=torch.int32, device="cuda")
        tg.fill_uniform_indices(t, n, bound, seed)
        assert np.array_equal(to_host(t), oracle.uniform_indices(n, bound, seed))


def test_run_indices_and_permutation_match_oracle(cuda):
    """The gather workload's index patterns, generated by the library, equal
    the oracle's generators (ragged last chunk included)."""
    torch = cuda
    for n, seed in [(32, 0), (33, 4), (100003, 2), (1 << 20, 7)]:
        t = torch.empty(n, dtype=torch.int32, device="cuda")
        tg.fill_run_indices(t, n, seed)
        assert np.array_equal(to_host(t), oracle.run_indices(n, seed))
    for n, seed in [(1, 0), (2, 5), (100003, 1), (1 << 20, 3)]:
        t = torch.empty(n, dtype=torch.int32, device="cuda")
        tg.fill_permutation(t, n, seed)
        assert np.array_equal(to_host(t), oracle.permutation(n, seed))
    with pytest.raises(tg.TroveError):
        tg.fill_run_indices(t, 31, 0)


def test_copy_host(cuda):
    torch = cuda
    for n, width, pinned in [(1, 12, False), (100003, 12, True), ((96 << 20) // 28 + 5, 28, True)]:
        src_h = torch.from_numpy(oracle.random_structs(n, width, seed=n).reshape(-1).copy())
        if pinned:
            src_h = src_h.pin_memory()
        dst_h = torch.zeros_like(src_h)
        if pinned:
            dst_h = dst_h.pin_memory()
        tg.copy_host(dst_h, src_h, n, width)
        assert torch.equal(dst_h, src_h)


def test_config1_contiguous_copy_12B(cuda):
    """N = 2^20 structs of 3 x uint32 (12 B), words from seed 0, through
    load/store_warp_contiguous (one launch, 256 threads per block), bit-exact
    against the CPU host loop."""
    torch = cuda
    n, width = 1 << 20, 12
    src_h = oracle.random_structs(n, width, seed=0)
    src = to_dev(torch, src_h)
    dst = torch.zeros_like(src)
    tg.copy(dst, src, n, width, path="warp")
    torch.cuda.synchronize()
    assert np.array_equal(to_host(dst), oracle.copy(src_h, n, width))


@pytest.mark.parametrize("width", WIDTHS)
def test_aos_soa_round_trip(cuda, width):
    torch = cuda
    s = width // 4
    for n in [1, 33, 4097, 100003]:
        aos_h = oracle.random_structs(n, width, seed=width + 7 * n)
        soa_expect = oracle.aos_to_soa(aos_h, n, s)
        assert np.array_equal(soa_expect.reshape(s, n), aos_h.view(np.uint32).reshape(n, s).T)
        aos = to_dev(torch, aos_h)
        for unroll, grid in [(0, 0), (1, 0), (2, 0), (4, 0), (8, 0), (2, -1), (1, 7)]:
            soa = torch.empty(n * width, dtype=torch.uint8, device="cuda")
            tg.aos_to_soa(soa, aos, n, width, unroll=unroll, grid=grid)
            assert np.array_equal(to_host(soa).view(np.uint32), soa_expect), (width, n, unroll, grid)
            back = torch.zeros_like(aos)
            tg.soa_to_aos(back, soa, n, width, unroll=unroll, grid=grid)
            assert np.array_equal(to_host(back), aos_h.reshape(-1)), (width, n, unroll, grid)


@pytest.mark.parametrize("width", [68, 96, 128, 132, 200, 256])
def test_index_ops_wide_structs(cuda, width):
    """Widths above 64 bytes: row-form kernels with a run-time word count."""
    torch = cuda
    n = 3000
    src_h = oracle.random_structs(n, width, seed=width)
    src = to_dev(torch, src_h)
    init = np.full(n * width, SENTINEL, np.uint8)
    for name, idx_h in index_sets(n, seed=width).items():
        idx = torch.from_numpy(idx_h).cuda()
        for path in ["auto", "warp"]:
            dst = to_dev(torch, init)
            tg.gather(dst, src, n, idx, n, width, path=path)
            assert np.array_equal(to_host(dst), oracle.gather(init, src_h, idx_h, n, width)), (name, path)
        if name in ("perm", "identity"):
            dst = to_dev(torch, init)
            tg.scatter(dst, n, src, idx, n, width)
            assert np.array_equal(to_host(dst), oracle.scatter(init, src_h, idx_h, n, width)), name
    bad = oracle.uniform_indices(n, n, 1).copy()
    bad[::7] = -3
    dst = to_dev(torch, init)
    tg.gather(dst, src, n, torch.from_numpy(bad).cuda(), n, width)
    e = init.reshape(n, width).copy()
    ok = bad >= 0
    e[ok] = src_h[bad[ok]]
    assert np.array_equal(to_host(dst), e.reshape(-1))


@pytest.mark.parametrize("width", WIDTHS)
def test_index_ops_default_route(cuda, width):
    """The one-chunk row-form kernels as a plain call takes them: the last
    struct of a chunk, the length where the unroll changes (2^16), a source
    longer and one shorter than the indices, and out-of-range indices at
    every position of a chunk."""
    torch = cuda
    for n, bound in [(1, 1), (31, 40), (65, 33), ((1 << 16), 5000), ((1 << 16) + 1, 70001), ((1 << 16) + 300, 1 << 16)]:
        src_h = oracle.random_structs(max(n, bound), width, seed=width + n)
        idx_h = oracle.uniform_indices(n, bound, n + 5).copy()
        idx_h[::37] = [-1, bound, 0x7FFFFFFF, -0x80000000][n % 4]
        ok = (idx_h >= 0) & (idx_h < bound)
        expect = np.full((n, width), SENTINEL, np.uint8)
        expect[ok] = src_h[idx_h[ok]]
        src = to_dev(torch, src_h)
        idx = torch.from_numpy(idx_h).cuda()
        buf, start = guarded(torch, n * width)
        tg.gather(buf[start:], src, bound, idx, n, width)
        assert np.array_equal(check_guards(buf, start, n * width), expect.reshape(-1)), ("gather", n, bound)
        perm_h = oracle.permutation(max(n, bound), 7)[:n].copy()
        perm_h[::41] = bound + 1 if bound < n else -7
        ok = (perm_h >= 0) & (perm_h < bound)
        expect = np.full((bound, width), SENTINEL, np.uint8)
        expect[perm_h[ok]] = src_h[:n][ok]
        buf, start = guarded(torch, bound * width)
        tg.scatter(buf[start:], bound, src, torch.from_numpy(perm_h).cuda(), n, width)
        assert np.array_equal(check_guards(buf, start, bound * width), expect.reshape(-1)), ("scatter", n, bound)


@pytest.mark.parametrize("width,offset", [(4, 0), (8, 0), (12, 0), (28, 4), (32, 16), (36, 0), (48, 0), (60, 8)])
def test_scatter_in_parts(cuda, width, offset):
    """Scatters onto destinations that take two parts (64 MiB and a little
    more) and one (just above 22 MiB): random and sorted indices, skipped ones
    among them, a last slab of one struct, rows that nothing is written to."""
    torch = cuda
    for bound in ((64 << 20) // width + 77, (22 << 20) // width + 1):
        n = (bound - 5) // 4096 * 4096 + 1
        src_h = oracle.random_structs(n, width, seed=width)
        src = torch.zeros(n * width + 64, dtype=torch.uint8, device="cuda")
        src[offset:offset + n * width] = to_dev(torch, src_h)
        perm = oracle.permutation(bound, width + 9)[:n].copy()
        for idx_h in (perm, np.sort(perm)):
            idx_h = idx_h.copy()
            idx_h[::4099] = -1
            idx_h[7::8191] = bound
            ok = (idx_h >= 0) & (idx_h < bound)
            expect = np.full((bound, width), SENTINEL, np.uint8)
            expect[idx_h[ok]] = src_h[ok]
            idx = torch.from_numpy(idx_h).cuda()
            for kw in ({}, {"path": "warp", "policy": 6}):
                buf, start = guarded(torch, bound * width, offset=offset)
                tg.scatter(buf[start:], bound, src[offset:], idx, n, width, **kw)
                assert np.array_equal(check_guards(buf, start, bound * width), expect.reshape(-1)), (bound, kw)


@pytest.mark.parametrize("where", ["dst", "src", "idx"])
@pytest.mark.parametrize("width", [12, 80])
def test_scatter_with_host_memory_is_one_plain_pass(cuda, width, where):
    torch = cuda
    n = (1 << 21) + 3 if width == 80 else (65 << 20) // width
    src = torch.randint(0, 255, (n, width), dtype=torch.uint8)
    idx = torch.randperm(n).to(torch.int32)
    expect = torch.empty_like(src)
    expect[idx.long()] = src
    side = {"src": src, "idx": idx, "dst": torch.zeros_like(src)}
    side = {k: t.pin_memory() if k == where else t.cuda() for k, t in side.items()}

    def run():
        tg.scatter(side["dst"], n, side["src"], side["idx"], n, width)

    run()
    torch.cuda.synchronize()
    assert torch.equal(side["dst"].cpu(), expect)
    on_gpu = {k: t.cuda() for k, t in side.items()}
    assert len(launched_grids(torch, run)) == 1
    rows = launched_grids(torch, run)[0]
    passes = launched_grids(torch, lambda: tg.scatter(on_gpu["dst"], n, on_gpu["src"], on_gpu["idx"], n, width))
    assert passes != [rows]


@pytest.mark.parametrize("src_at,dst_at", [(4, 0), (8, 4), (1, 0)])
def test_copy_to_host_memory_between_alignments(cuda, src_at, dst_at):
    torch = cuda
    nbytes = (1 << 20) + 5
    src = torch.randint(0, 255, (nbytes + 64,), dtype=torch.uint8, device="cuda")
    dst = torch.zeros(nbytes + 64, dtype=torch.uint8).pin_memory()
    tg.copy(dst.data_ptr() + dst_at, src.data_ptr() + src_at, nbytes, 1)
    torch.cuda.synchronize()
    assert torch.equal(dst[dst_at:dst_at + nbytes], src[src_at:src_at + nbytes].cpu())
    assert not dst[:dst_at].any() and not dst[dst_at + nbytes:].any()


@pytest.mark.parametrize("mib", [41, 65, 130])
@pytest.mark.parametrize("width", [8, 12, 24, 36, 48, 72, 13])
def test_scatter_orders_of_indices(cuda, width, mib):
    """Destinations that are fetched first and ones in two or more parts, with rows
    in order, in shuffled runs, at random, at random within a tenth of the destination
    (one part, or less than L2 holds) and few valid ones: whichever form the sample of
    the indices picks, every valid row arrives and nothing else changes."""
    torch = cuda
    bound = (mib << 20) // width
    n = bound - 3
    src = torch.randint(0, 255, (n, width), dtype=torch.uint8, device="cuda")
    order = torch.arange(n, device="cuda")
    runs = (torch.randperm(n // 32, device="cuda")[:, None] * 32 + torch.arange(32, device="cuda")).reshape(-1)
    tenth = bound // 10
    inside = torch.full((n,), -1, device="cuda", dtype=torch.int64)
    inside[torch.randperm(n, device="cuda")[:tenth]] = torch.randperm(tenth, device="cuda") + bound // 2
    wide = torch.full((n,), -1, device="cuda", dtype=torch.int64)
    wide[::3] = (torch.randperm(bound // 2, device="cuda") + bound // 4)[:(n + 2) // 3]
    few = torch.full((n,), bound, device="cuda", dtype=torch.int64)
    few[7] = bound - 1
    tenths = torch.where(torch.rand(n, device="cuda") < 0.9, torch.full_like(order, bound), torch.randperm(bound, device="cuda")[:n])
    for name, idx in (("order", order), ("runs", torch.cat([runs, order[runs.numel():]])),
                      ("random", torch.randperm(bound, device="cuda")[:n]), ("inside", inside), ("wide", wide),
                      ("few", few), ("tenths", tenths), ("tenths in order", torch.where(tenths < bound, order, tenths))):
        idx = idx.to(torch.int32)
        ok = (idx >= 0) & (idx < bound)
        expect = torch.full((bound, width), SENTINEL, dtype=torch.uint8, device="cuda")
        expect[idx[ok].long()] = src[ok]
        dst = torch.full((bound, width), SENTINEL, dtype=torch.uint8, device="cuda")
        tg.scatter(dst, bound, src, idx, n, width)
        assert torch.equal(dst, expect), name


@pytest.mark.parametrize("width", [12, 36, 48, 68])
@pytest.mark.parametrize("grid,unroll", [(1, 0), (37, 2), (-1, 1)])
def test_scatter_in_parts_on_a_requested_grid(cuda, width, grid, unroll):
    """Policy 6 onto a little more than 128 MiB: what is launched is that grid, and
    the rows arrive as on the default one."""
    torch = cuda
    bound = (128 << 20) // width + 1
    n = (1 << 16) + 3 if grid == 1 else bound - 2
    if grid == 1:
        bound = 2 * n  # a few blocks: small enough to stay quick, one pass
    src = torch.randint(0, 255, (n, width), dtype=torch.uint8, device="cuda")
    idx = torch.randperm(bound, device="cuda")[:n].to(torch.int32)
    idx[5], idx[n - 1] = -1, bound
    ok = (idx >= 0) & (idx < bound)
    expect = torch.full((bound, width), SENTINEL, dtype=torch.uint8, device="cuda")
    expect[idx[ok].long()] = src[ok]
    dst = torch.full((bound, width), SENTINEL, dtype=torch.uint8, device="cuda")

    def run():
        tg.scatter(dst, bound, src, idx, n, width, path="warp", policy=6, grid=grid,
                   unroll=unroll if width <= 64 else 0)

    run()
    assert torch.equal(dst, expect)
    grids = launched_grids(torch, run)
    assert len(set(grids)) == 1 and (grid < 0 or grids[0] == grid), grids


@pytest.mark.parametrize("n", [1, 2, 33, 4097])
def test_scatter_in_parts_short(cuda, n):
    """The same policy asked for on arrays of any size, onto one row too."""
    torch = cuda
    for width, bound in [(12, n), (20, n + 9), (4, 1)]:
        src_h = oracle.random_structs(n, width, seed=n)
        idx_h = oracle.permutation(n, 3) if bound >= n else np.where(np.arange(n) == n // 2, 0, -1).astype(np.int32)
        ok = (idx_h >= 0) & (idx_h < bound)
        expect = np.full((bound, width), SENTINEL, np.uint8)
        expect[idx_h[ok]] = src_h[ok]
        buf, start = guarded(torch, bound * width)
        tg.scatter(buf[start:], bound, to_dev(torch, src_h), torch.from_numpy(idx_h).cuda(), n, width, path="warp",
                   policy=6)
        assert np.array_equal(check_guards(buf, start, bound * width), expect.reshape(-1)), (n, width)


def test_default_stream_is_torchs_current_one(cuda):
    torch = cuda
    assert tg._stream(None) == torch.cuda.current_stream().cuda_stream
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert tg._stream(None) == side.cuda_stream != 0
    assert tg._stream(None) == torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("width", [5, 6, 7, 12, 13, 20, 31, 47, 64, 65, 217])
def test_index_ops_packed(cuda, width):
    """Rows of any width at any alignment: chunk and array ends, skipped rows,
    the lengths and widths where the route changes, source and destination at
    every offset from a word boundary; bytes around the arrays stay."""
    torch = cuda
    lengths = [1, 9, 33, 131, 70001] + ([(1 << 19) + 77] if width < 20 else [])
    for n in lengths:
        for bound in (n + 3, max(1, n - n // 3)):
            rows = max(n, bound)
            src_h = np.frombuffer(oracle.random_words((rows * width + 3) // 4, n).tobytes()[:rows * width], np.uint8)
            src_h = src_h.reshape(rows, width)
            uni = oracle.uniform_indices(n, bound, n + 1).copy()
            perm = oracle.permutation(rows, 3)[:n].copy()
            for soff, doff in [(1, 0), (0, 3), (2, 1), (3, 2)] if n < 1000 else [(1, 3)]:
                src = torch.zeros(rows * width + 8, dtype=torch.uint8, device="cuda")
                src[soff:soff + rows * width] = to_dev(torch, src_h)
                for skip in (False, True):
                    if skip:
                        uni[::5] = -1
                        perm[::5] = bound
                    buf, start = guarded(torch, n * width, offset=doff)
                    tg.gather(buf[start:], src[soff:], bound, torch.from_numpy(uni).cuda(), n, width)
                    ok = uni >= 0
                    expect = np.full((n, width), SENTINEL, np.uint8)
                    expect[ok] = src_h[uni[ok]]
                    assert np.array_equal(check_guards(buf, start, n * width), expect.reshape(-1)), (n, bound, soff, doff)
                    buf, start = guarded(torch, bound * width, offset=doff)
                    tg.scatter(buf[start:], bound, src[soff:], torch.from_numpy(perm).cuda(), n, width)
                    ok = perm < bound
                    expect = np.full((bound, width), SENTINEL, np.uint8)
                    expect[perm[ok]] = src_h[:n][ok]
                    assert np.array_equal(check_guards(buf, start, bound * width), expect.reshape(-1)), (n, bound, soff,
                                                                                                         doff)


@pytest.mark.parametrize("width", [6, 7, 8, 9, 10, 11, 13, 30, 33, 47])
def test_index_ops_packed_orders_of_indices(cuda, width):
    """Rows in order, backwards, in shuffled runs, with most of them skipped, and all
    of these in one array: rows that go by bytes, by words, and by what the sample of
    the indices says."""
    torch = cuda
    for n in (100, 70003, (1 << 20) + 7):
        src = torch.randint(0, 255, (n * width + 8,), dtype=torch.uint8, device="cuda")
        rows = src[1:1 + n * width].view(n, width)
        order = torch.arange(n, device="cuda")
        few = torch.full((n,), -1, device="cuda", dtype=torch.int64)
        few[::11] = torch.randperm(n, device="cuda")[:few[::11].numel()]
        mixed = torch.randperm(n, device="cuda")
        mixed[n // 3:n // 2] = few[n // 3:n // 2]
        free = torch.ones(n, dtype=torch.bool, device="cuda")  # rows that mixed's first third does not name
        free[mixed[:n // 3]] = False
        mixed[n // 2:] = torch.where(free[order[n // 2:]], order[n // 2:], torch.full_like(order[n // 2:], n))
        for name, idx in (("order", order), ("back", order.flip(0)), ("few", few),
                          ("runs", torch.cat([(torch.randperm(n // 32, device="cuda")[:, None] * 32 + torch.arange(
                              32, device="cuda")).reshape(-1), order[n // 32 * 32:]])), ("mixed", mixed)):
            ok = (idx >= 0) & (idx < n)
            i32 = idx.to(torch.int32)
            expect = torch.full((n, width), SENTINEL, dtype=torch.uint8, device="cuda")
            expect[ok] = rows[idx[ok]]
            dst = torch.full((n * width + 8,), SENTINEL, dtype=torch.uint8, device="cuda")
            tg.gather(dst[3:], rows, n, i32, n, width)
            assert torch.equal(dst[3:3 + n * width].view(n, width), expect), ("gather", n, name)
            assert bool((dst[:3] == SENTINEL).all()) and bool((dst[3 + n * width:] == SENTINEL).all())
            if name == "mixed":  # no row twice: few's part may repeat one of the others
                seen = torch.zeros(n + 1, dtype=torch.bool, device="cuda")
                seen[torch.cat([idx[:n // 3], idx[n // 2:]])] = True
                mid = idx[n // 3:n // 2]
                idx = idx.clone()
                idx[n // 3:n // 2] = torch.where((mid >= 0) & ~seen[mid.clamp(min=0)], mid, torch.full_like(mid, -1))
                ok = (idx >= 0) & (idx < n)
                i32 = idx.to(torch.int32)
            expect = torch.full((n, width), SENTINEL, dtype=torch.uint8, device="cuda")
            expect[idx[ok]] = rows[ok]
            dst = torch.full((n * width + 8,), SENTINEL, dtype=torch.uint8, device="cuda")
            tg.scatter(dst[2:], n, rows, i32, n, width)
            assert torch.equal(dst[2:2 + n * width].view(n, width), expect), ("scatter", n, name)
            assert bool((dst[:2] == SENTINEL).all()) and bool((dst[2 + n * width:] == SENTINEL).all())


@pytest.mark.parametrize("width,n", [(7, 65537), (7, 524291), (7, 1 << 20), (13, 32767), (13, 32768), (13, 131073),
                                     (13, 786439), (13, 3145729), (29, 49153), (29, 1048577), (47, 131071), (47, 131072), (47, 524291),
                                     (47, 2097153), (111, 393217), (111, 1048579), (217, 393216), (217, 393215)])
def test_index_ops_packed_rows_to_a_warp(cuda, width, n):
    """Packed rows at the lengths where the rows to a warp change: every chunk
    size with a remainder, skipped rows, arrays at odd addresses."""
    torch = cuda
    raw = torch.zeros(n * width + 64, dtype=torch.uint8, device="cuda")
    tg.fill_random_u32(raw, raw.numel() // 4, seed=width)
    src = raw[3:3 + n * width]
    perm = torch.empty(n, dtype=torch.int32, device="cuda")
    tg.fill_permutation(perm, n, 5)
    perm[::7] = -1
    ok = perm >= 0
    rows = src.view(n, width)
    for scatter in (False, True):
        buf = torch.full((n * width + 32,), SENTINEL, dtype=torch.uint8, device="cuda")
        dst = buf[17:17 + n * width]
        expect = torch.full((n, width), SENTINEL, dtype=torch.uint8, device="cuda")
        if scatter:
            tg.scatter(dst, n, src, perm, n, width)
            expect[perm[ok].long()] = rows[ok]
        else:
            tg.gather(dst, src, n, perm, n, width)
            expect[ok] = rows[perm[ok].long()]
        assert torch.equal(dst.view(n, width), expect), scatter
        assert bool((buf[:17] == SENTINEL).all()) and bool((buf[17 + n * width:] == SENTINEL).all()), scatter


@pytest.mark.parametrize("shift", range(1, 16))
def test_copy_between_alignments(cuda, shift):
    """Copies whose two addresses differ modulo 16, on both sides of the length
    from which they are joined from aligned vectors, at lengths that end
    anywhere in a vector; bytes around the destination stay."""
    torch = cuda
    n = (512 << 10) + 40
    src_h = np.frombuffer(oracle.random_words(n // 4 + 16, shift).tobytes(), np.uint8)
    src = to_dev(torch, src_h)
    for nbytes in [(512 << 10) - 1, 512 << 10, (512 << 10) + shift, n]:
        for doff in (0, 5, 16 - shift, 15):
            soff = (doff + shift) % 16
            for kw in ({}, {"path": "vector", "unroll": 2}, {"path": "vector", "unroll": 8, "grid": 3}):
                buf, start = guarded(torch, nbytes, offset=doff)
                tg.copy(buf[start:], src[soff:], nbytes, 1, **kw)
                assert np.array_equal(check_guards(buf, start, nbytes), src_h[soff:soff + nbytes]), (nbytes, doff, kw)


@pytest.mark.parametrize("offset", [0, 3, 15])
def test_copy_equal_alignment_short(cuda, offset):
    """Copies whose addresses agree modulo 16, around the length up to which
    a thread takes one vector; bytes around the destination stay."""
    torch = cuda
    n = (1 << 20) + 40
    src_h = np.frombuffer(oracle.random_words(n // 4 + 16, offset).tobytes(), np.uint8)
    src = to_dev(torch, src_h)
    for nbytes in (16 - offset, 17, 4096 - offset, 4097, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, n):
        buf, start = guarded(torch, nbytes, offset=offset)
        tg.copy(buf[start:], src[offset:], nbytes, 1)
        assert np.array_equal(check_guards(buf, start, nbytes), src_h[offset:offset + nbytes]), nbytes


@pytest.mark.parametrize("width,offset", [(68, 0), (68, 4), (80, 0), (96, 8), (132, 0), (200, 0), (256, 0), (1028, 0)])
def test_index_ops_wide_default_route(cuda, width, offset):
    """Rows wider than 64 bytes as a plain call takes them, at the lengths where
    the rows to a warp change, at every word size, with skipped rows."""
    torch = cuda
    for n in [1, 3, 5, 1 << 13, (1 << 13) + 1, (1 << 15) + 3] + ([(1 << 16) + 5, (1 << 17) + 9] if width < 100 else []):
        bound = n + 7
        src_h = oracle.random_structs(bound, width, seed=n)
        src = torch.zeros(bound * width + 64, dtype=torch.uint8, device="cuda")
        src[offset:offset + bound * width] = to_dev(torch, src_h)
        perm = oracle.permutation(bound, n)[:n].copy()
        perm[n // 2:n // 2 + 1] = -1
        perm[::11] = bound
        ok = (perm >= 0) & (perm < bound)
        idx = torch.from_numpy(perm).cuda()
        expect = np.full((n, width), SENTINEL, np.uint8)
        expect[ok] = src_h[perm[ok]]
        buf, start = guarded(torch, n * width, offset=offset)
        tg.gather(buf[start:], src[offset:], bound, idx, n, width)
        assert np.array_equal(check_guards(buf, start, n * width), expect.reshape(-1)), ("gather", n)
        expect = np.full((bound, width), SENTINEL, np.uint8)
        expect[perm[ok]] = src_h[:n][ok]
        buf, start = guarded(torch, bound * width, offset=offset)
        tg.scatter(buf[start:], bound, src[offset:], idx, n, width)
        assert np.array_equal(check_guards(buf, start, bound * width), expect.reshape(-1)), ("scatter", n)


def test_scatter_wide_rows_in_parts(cuda):
    """2^21 rows and more wider than 64 bytes go in parts: the sorted and the
    random form, and 4-byte words."""
    torch = cuda
    n, width = (1 << 21) + 3, 68
    src = torch.randint(0, 255, (n, width), dtype=torch.uint8, device="cuda")
    for idx in (torch.randperm(n, device="cuda").to(torch.int32), torch.arange(n, device="cuda", dtype=torch.int32)):
        idx[5] = -1
        idx[n - 1] = n
        ok = (idx >= 0) & (idx < n)
        expect = torch.full((n, width), SENTINEL, dtype=torch.uint8, device="cuda")
        expect[idx[ok].long()] = src[ok]
        dst = torch.full((n, width), SENTINEL, dtype=torch.uint8, device="cuda")
        tg.scatter(dst, n, src, idx, n, width)
        assert torch.equal(dst, expect)


@pytest.mark.parametrize("width", [(34 << 20) + 4, (8 << 20) + 4, 8 << 20])
def test_scatter_rows_of_many_mebibytes_with_parts_asked_for(cuda, width):
    """Rows so wide that the last ones of 512 lie beyond 4 GiB of 4-byte words' worth
    of offset, and rows around the widest that go in parts: the row named by the one
    valid index arrives, the others stay."""
    torch = cuda
    n, bound = 512, (64 << 20) // width + 2
    src = torch.empty(n * width, dtype=torch.uint8, device="cuda")
    row = torch.randint(0, 255, (width,), dtype=torch.uint8, device="cuda")
    for at in (510, 3):
        src[at * width:(at + 1) * width] = row
        idx = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        idx[at] = bound - 1
        dst = torch.full((bound * width,), SENTINEL, dtype=torch.uint8, device="cuda")
        tg.scatter(dst, bound, src, idx, n, width, path="warp", policy=6)
        assert torch.equal(dst[(bound - 1) * width:], row)
        assert bool((dst[:(bound - 1) * width] == SENTINEL).all())


@pytest.mark.parametrize("width", [8, 44])
@pytest.mark.parametrize("modulus", [1, 2, 3, 6, 625, 640, 1 << 31, (1 << 31) + 1, 0xFFFFFFFE, 0xFFFFFFFF])
def test_copy_exit_moduli(cuda, modulus, width):
    """The exit predicate for odd, even, power-of-two and largest moduli, on words
    around every kind of multiple: the smallest, the largest, the wrap-around."""
    torch = cuda
    n = 40000
    words = oracle.random_words(width // 4 * n, modulus & 0xFFFF).astype(np.uint32).copy()
    first = words[::width // 4]
    edge = np.array([0, 1, modulus - 2, modulus - 1, modulus, 2 * modulus - 1, 0xFFFFFFFF, 0xFFFFFFFE, 1 << 31]) & 0xFFFFFFFF
    first[0:18:2] = edge.astype(np.uint32)
    near = (first[2000:4000].astype(np.uint64) // modulus) * modulus + modulus - 1
    first[2000:4000] = (near & 0xFFFFFFFF).astype(np.uint32)
    src_h = words.view(np.uint8).reshape(n, width)
    init = np.full(n * width, SENTINEL, np.uint8)
    expect, _ = oracle.copy_exit(init, src_h, n, width, modulus)
    for path in ("warp", "block"):
        dst = to_dev(torch, init)
        tg.copy_exit(dst, to_dev(torch, src_h), n, width, modulus, path=path)
        assert np.array_equal(to_host(dst), expect), (modulus, path)
