"""Parity of the GPU partitioner with the oracle / reference goldens, through the C ABI."""
import ctypes

import numpy as np
import pytest

from conftest import kat_indptr, sha256_block4, require_cuda
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_golden_block4_files_bit_exact_host_entry(kat):
    from accelgcn import partition
    require_cuda()
    for name, entry in kat.items():
        got = partition.block_level_partition(kat_indptr(entry))
        assert len(got) == entry["n_blocks"], name
        assert sha256_block4(got) == entry["sha256"], name


def test_golden_block4_files_bit_exact_device_entry(kat):
    import torch
    from accelgcn import partition
    dev = require_cuda()
    for name in ("pubmed", "am", "citation", "ppa", "arxiv", "youtube"):
        ip = torch.from_numpy(kat_indptr(kat[name])).to(dev)
        got = partition.block_level_partition_device(ip).cpu().numpy()
        assert sha256_block4(got) == kat[name]["sha256"], name


def test_reference_script_edge_cases_bit_exact(edge_cases):
    from accelgcn import partition
    require_cuda()
    for name, (indptr, want) in edge_cases.items():
        got = partition.block_level_partition(indptr)
        assert np.array_equal(got, want), name


@pytest.mark.parametrize("seed", range(8))
def test_random_degree_sequences_match_oracle(seed):
    from accelgcn import partition
    require_cuda()
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 200_000))
    pool = np.array([0, 0, 1, 1, 1, 2, 3, 12, 31, 32, 33, 64, 65, 96, 97, 128, 129, 191, 192, 383, 384, 385, 769, 4000])
    if seed % 2:
        deg = rng.choice(pool, n)                         # unsorted, many short runs
    else:
        deg = np.sort(rng.choice(pool, n))                # sorted, long runs crossing many tiles
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    assert np.array_equal(partition.block_level_partition(indptr), oracle.partition(indptr))


def test_nonzero_first_pointer_and_all_zero_degrees():
    from accelgcn import partition
    require_cuda()
    deg = np.array([3, 3, 3, 0, 500])
    ip = (np.concatenate([[0], np.cumsum(deg)]) + 17).astype(np.int32)
    assert np.array_equal(partition.block_level_partition(ip), oracle.partition(ip - 17))
    # a graph with rows but no nonzero: no tuples (the reference script fails inside scipy here)
    assert partition.block_level_partition(np.zeros(9, dtype=np.int32)).shape == (0, 4)


def test_full_size_degree_sequence_matches_oracle_and_invariants():
    # 5 million rows with the degree mix of the large configurations: bit-exact against the C
    # oracle, plus format invariants that hold at any size
    from accelgcn import partition
    require_cuda()
    rng = np.random.default_rng(99)
    n = 5_000_000
    deg = np.sort(np.minimum((rng.pareto(1.2, n) * 6).astype(np.int64), 20_000))
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    got = partition.block_level_partition(indptr)
    assert np.array_equal(got, oracle.partition(indptr))
    d, row, loc, info = got.T.astype(np.int64)
    small = d <= 384
    nz = np.where(small, (info & 0xFFFF) * d, info)
    assert nz.sum() == indptr[-1] and np.all(nz <= 384)
    assert np.array_equal(loc, np.concatenate([[0], np.cumsum(nz)[:-1]]))        # tuples tile the nonzeros
    assert np.array_equal(loc[small], indptr[row[small]])


def test_error_behaviour():
    from accelgcn import _lib
    require_cuda()
    lib = _lib.load()
    n = ctypes.c_int64(0)
    bad = np.array([0, 5, 3, 9], dtype=np.int32)                                  # negative degree
    assert lib.agcn_partition_host(bad.ctypes.data, 3, None, 0, ctypes.byref(n)) == _lib.ERR_RANGE
    ip = np.array([0, 1, 2, 1000], dtype=np.int32)
    out = np.zeros((2, 4), dtype=np.int32)
    assert lib.agcn_partition_host(ip.ctypes.data, 3, out.ctypes.data, 2, ctypes.byref(n)) == _lib.ERR_CAPACITY
    assert n.value == 4                                                           # 1 + ceil(998 / 384)


def test_drop_in_script_same_files_as_the_reference(kat, tmp_path):
    # run like the reference script: cwd holding ./graphs/<g>.config + .new_indptr -> ./block_level_meta/<g>.block4
    import subprocess, sys, os
    from conftest import PKG
    require_cuda()
    os.makedirs(tmp_path / "graphs")
    for name in ("pubmed", "collab"):
        (tmp_path / "graphs" / f"{name}.config").write_text("")
        kat_indptr(kat[name]).tofile(tmp_path / "graphs" / f"{name}.new_indptr")
    subprocess.check_call([sys.executable, os.path.join(PKG, "block_level_partition.py")], cwd=tmp_path,
                          stdout=subprocess.DEVNULL)
    for name in ("pubmed", "collab"):
        got = np.fromfile(tmp_path / "block_level_meta" / f"{name}.block4", dtype=np.int32)
        assert sha256_block4(got) == kat[name]["sha256"], name


@pytest.mark.parametrize("run", [1, 2047, 2048, 2049, 6144, 5000])
def test_runs_across_tiles_match_oracle(run):
    # tiles of 2048 rows: a run that begins before a tile decides which of the tile's leading rows open a tuple
    import torch
    from accelgcn import partition
    dev = require_cuda()
    # the last: 391 thousand tuples in the run's rows, many tiles of more than 4096
    for degs in ([1, 40, 70, 100, 150, 300, 385], [0, 7], [33, 0, 33, 500], [2, 150_000_000 // run, 3]):
        indptr = np.concatenate([[0], np.cumsum(np.repeat(degs, run))]).astype(np.int32)
        want = oracle.partition(indptr)
        assert np.array_equal(partition.block_level_partition(indptr), want)
        assert np.array_equal(partition.block_level_partition_device(torch.from_numpy(indptr).to(dev)).cpu().numpy(), want)


@pytest.mark.parametrize("rows", [3_000, 600_000])
@pytest.mark.parametrize("total", [4095, 4096, 4097, 8192, 30_000])
def test_tiles_of_many_tuples_match_oracle(rows, total):
    # a tile (2048 rows) of more than 4096 tuples is written by several blocks, 4096 output positions each: hub rows that
    # make up `total` tuples between rows of one and of none, at the start, at the end and in neighbouring tiles; few tiles,
    # and more than the 256 that the scan of the tiles takes at a time (the first tile has exactly `total` tuples)
    import torch
    from accelgcn import partition
    dev = require_cuda()
    rng = np.random.default_rng(total)
    deg = rng.choice([0, 1, 5, 40, 200, 384], rows)
    for first in (0, 2047, rows - 900):
        hubs = 1 + rng.multinomial(total - 700, rng.dirichlet(np.ones(700)))
        deg[first:first + 700] = hubs * 384 - rng.integers(0, 300, 700)
    deg[700:2048] = 0
    deg[4096:8192] = 0                                  # tiles without any tuple
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    want = oracle.partition(indptr)
    assert np.array_equal(partition.block_level_partition(indptr), want)
    assert np.array_equal(partition.block_level_partition_device(torch.from_numpy(indptr).to(dev)).cpu().numpy(), want)


@pytest.mark.parametrize("n", [5_000, 700_000])
def test_on_another_stream_the_tuples_are_complete_on_return(n):
    # with a stream that is not the current one the caller goes on elsewhere, here while that stream is kept busy; few tiles
    # of 2048 rows, and more than the 256 that their scan takes at a time
    import torch
    from accelgcn import partition
    dev = require_cuda()
    indptr = np.concatenate([[0], np.cumsum(np.sort(np.random.default_rng(n).integers(0, 60, n)))]).astype(np.int32)
    want = oracle.partition(indptr)
    side = torch.cuda.Stream(dev)
    busy = torch.zeros(1 << 26, device=dev)
    for _ in range(4):
        d_ip = torch.from_numpy(indptr).to(dev)
        torch.cuda.synchronize()
        out = partition.block_level_partition_device(d_ip, stream=side)
        assert side.query()                       # nothing of the call is left on that stream
        d_ip.zero_()                              # the row pointers are the caller's again
        assert np.array_equal(out.cpu().numpy(), want)
        with torch.cuda.stream(side):
            busy.add_(1)


@pytest.mark.parametrize("n", [5_000, 2_048 * 256, 2_048 * 256 + 1, 700_000])
def test_row_pointers_may_be_overwritten_behind_the_call_on_its_stream(n):
    # the tuples are written behind the call, from the row pointers; work behind it on the same stream comes later.  The
    # scan of the tiles takes 256 at a time: one round of it, exactly, and a second one of a single row
    import torch
    from accelgcn import partition
    dev = require_cuda()
    indptr = np.concatenate([[0], np.cumsum(np.sort(np.random.default_rng(n).integers(0, 60, n)))]).astype(np.int32)
    want = oracle.partition(indptr)
    src = torch.from_numpy(indptr).to(dev)
    for _ in range(4):
        d_ip = src.clone()
        out = partition.block_level_partition_device(d_ip)
        d_ip.fill_(7)
        del d_ip
        torch.full((n + 1,), -1, dtype=torch.int32, device=dev)          # takes the block that was just given back
        assert np.array_equal(out.cpu().numpy(), want)


def test_count_does_not_depend_on_what_the_scratch_held():
    # the scratch is pool memory, never cleared: here, before every call, the pool's block of that size is filled (as the
    # row pointers of a call that is refused) with descriptions of 300 tiles and marks that say that they are there, as a
    # kernel that looked for marks in this memory left and expected them.  Own process: the marks count its calls.  Of the
    # row pointers the last tile's are in L2, so that it is described before the others.
    import subprocess, sys
    from conftest import PKG
    require_cuda()
    code = """
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import torch
from accelgcn import _lib
lib = _lib.load()
tiles, rows = 300, 2048 * 300
d_ip = torch.arange(rows + 1, dtype=torch.int32, device="cuda")
flush = torch.empty(1 << 26, device="cuda")
n = ctypes.c_int64(0)
for k in range(60):
    held = np.zeros(2816, dtype=np.int32)
    held[:4 * tiles].reshape(tiles, 4)[:] = (-1, 0, 0, 1_000_000)          # last run start, two of leading rows, tuples
    held[1216:1216 + 2 * tiles].reshape(tiles, 2)[:] = (2 * k + 2, 0x7ff4a9c3)
    assert lib.agcn_partition_host(held.ctypes.data, len(held) - 1, None, 0, ctypes.byref(n)) == _lib.ERR_RANGE
    flush.zero_()
    d_ip[-5000:].sum()
    torch.cuda.synchronize()
    _lib.check(lib.agcn_partition_device(d_ip.data_ptr(), rows, None, 0, ctypes.byref(n), None))
    assert n.value == rows // 12, (k, n.value)
"""
    out = subprocess.run([sys.executable, "-c", code, PKG], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]


def test_many_calls_at_once():
    # 70 calls under way together, six more than there are arrival counters: each on a stream of its own that is kept
    # busy until all have been started; twice, so that counters are used again
    import threading
    import torch
    from accelgcn import _lib
    dev = require_cuda()
    lib = _lib.load()
    rng = np.random.default_rng(5)
    sizes = [int(n) for n in rng.integers(1, 40_000, 70)]
    ips = [np.concatenate([[0], np.cumsum(rng.integers(0, 500, n))]).astype(np.int32) for n in sizes]
    want = [oracle.partition(ip) for ip in ips]
    d_ips = [torch.from_numpy(ip).to(dev) for ip in ips]
    outs = [torch.full((len(w) + 1, 4), -7, dtype=torch.int32, device=dev) for w in want]
    streams = [torch.cuda.Stream(dev) for _ in sizes]
    answers = [None] * len(sizes)

    def one(k):
        n = ctypes.c_int64(0)
        rc = lib.agcn_partition_device(d_ips[k].data_ptr(), sizes[k], outs[k].data_ptr(), len(want[k]), ctypes.byref(n), streams[k].cuda_stream)
        answers[k] = (rc, n.value)

    for _ in range(2):
        for o in outs:
            o.fill_(-7)
        torch.cuda.synchronize()
        for s in streams:
            with torch.cuda.stream(s):
                torch.cuda._sleep(100_000_000)
        threads = [threading.Thread(target=one, args=(k,)) for k in range(len(sizes))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k, w in enumerate(want):
            assert answers[k] == (0, len(w)), k
            got = outs[k].cpu().numpy()
            assert np.array_equal(got[:-1], w) and (got[-1] == -7).all(), k
