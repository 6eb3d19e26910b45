"""GPU degree sort + CSR permute against the CPU oracle (stable ascending argsort)."""
import numpy as np
import pytest

from conftest import require_cuda
from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(g, relabel):
    from accelgcn import degree_sort
    ip, ix, v = g.indptr.numpy(), g.indices.numpy(), g.vals.numpy()
    got = degree_sort.degree_sort(ip, ix, v, relabel_cols=relabel)
    want = oracle.degree_sort(ip, ix, v, relabel_cols=relabel)
    for a, b, what in zip(got, want, ("perm", "indptr", "indices", "vals")):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("cfg,scale", [(1, 1.0), (2, 0.01), (3, 0.02), (4, 0.05), (5, 0.001)])
@pytest.mark.parametrize("relabel", [False, True])
def test_matches_oracle_on_synthetic_configs(cfg, scale, relabel):
    from accelgcn import synth
    require_cuda()
    _check(synth.make_config(cfg, "cpu", scale), relabel)


def test_device_entry_and_properties_at_scale():
    # 2 million rows, degrees up to 2^17 (three radix passes): oracle equality for the
    # permutation, then properties of the permuted matrix
    import torch
    from accelgcn import degree_sort
    dev = require_cuda()
    rng = np.random.default_rng(5)
    n = 2_000_000
    deg = np.minimum((rng.pareto(1.1, n) * 3).astype(np.int64), 130_000)
    deg[rng.integers(0, n, 3)] = [70_000, 131_000, 66_000]
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    assert indptr[-1] < 2**31
    nnz = int(indptr[-1])
    idx = rng.integers(0, n, nnz, dtype=np.int32)
    val = rng.random(nnz, dtype=np.float32)
    t_ip = torch.from_numpy(indptr.astype(np.int32)).to(dev)
    perm, nip, nix, nv = degree_sort.degree_sort_device(t_ip, torch.from_numpy(idx).to(dev),
                                                        torch.from_numpy(val).to(dev), relabel_cols=True)
    perm, nip = perm.cpu().numpy(), nip.cpu().numpy()
    assert np.array_equal(perm, np.argsort(deg, kind="stable"))
    assert np.array_equal(np.diff(nip.astype(np.int64)), deg[perm])
    inv = np.empty(n, dtype=np.int64); inv[perm] = np.arange(n)
    nix, nv = nix.cpu().numpy(), nv.cpu().numpy()
    for r in rng.integers(0, n, 200).tolist() + [n - 1, n - 2, n - 3]:
        o = perm[r]
        assert np.array_equal(nix[nip[r]:nip[r + 1]], inv[idx[indptr[o]:indptr[o + 1]]])
        assert np.array_equal(nv[nip[r]:nip[r + 1]], val[indptr[o]:indptr[o + 1]])
    assert np.isclose(float(nv.astype(np.float64).sum()), float(val.astype(np.float64).sum()), rtol=1e-9)


def test_all_rows_empty_and_single_row():
    from accelgcn import degree_sort
    require_cuda()
    perm, nip, nix, _ = degree_sort.degree_sort(np.zeros(6, dtype=np.int32), np.zeros(0, dtype=np.int32))
    assert perm.tolist() == [0, 1, 2, 3, 4] and nip.tolist() == [0] * 6 and len(nix) == 0
    perm, nip, nix, _ = degree_sort.degree_sort(np.array([0, 3], dtype=np.int32), np.array([0, 0, 0], dtype=np.int32))
    assert perm.tolist() == [0] and nip.tolist() == [0, 3] and nix.tolist() == [0, 0, 0]


def test_bad_input_is_an_error_not_a_fault():
    from accelgcn import degree_sort, AccelGcnError
    require_cuda()
    with pytest.raises(AccelGcnError):
        degree_sort.degree_sort(np.array([0, 2, 1], dtype=np.int32), np.array([0, 1], dtype=np.int32))
    with pytest.raises(AccelGcnError):       # column 9 cannot be relabelled in a 2-row matrix
        degree_sort.degree_sort(np.array([0, 1, 2], dtype=np.int32), np.array([0, 9], dtype=np.int32), relabel_cols=True)


def test_values_given_but_not_wanted_and_wrong_nnz():
    # the C ABI allows d_vals != NULL with d_new_vals == NULL (the values are simply not permuted),
    # and rejects an nnz that is not the matrix's own count instead of reading past the arrays
    import ctypes
    import torch
    from accelgcn import _lib, synth
    dev = require_cuda()
    lib = _lib.load()
    g = synth.make_config(1, dev, 0.25)
    n, nnz = g.n, g.nnz
    perm = torch.empty(n, dtype=torch.int32, device=dev)
    nip = torch.empty(n + 1, dtype=torch.int32, device=dev)
    nix = torch.full((nnz,), -1, dtype=torch.int32, device=dev)
    rc = lib.agcn_degree_sort_device(g.indptr.data_ptr(), g.indices.data_ptr(), g.vals.data_ptr(), n, nnz, 1,
                                     perm.data_ptr(), nip.data_ptr(), nix.data_ptr(), None, None)
    assert rc == _lib.OK, lib.agcn_last_error()
    torch.cuda.synchronize()
    want = oracle.degree_sort(g.indptr.cpu().numpy(), g.indices.cpu().numpy(), None, True)
    assert np.array_equal(perm.cpu().numpy(), want[0]) and np.array_equal(nix.cpu().numpy(), want[2])
    for wrong in (nnz + 4096, nnz - 1):
        rc = lib.agcn_degree_sort_device(g.indptr.data_ptr(), g.indices.data_ptr(), None, n, wrong, 0,
                                         perm.data_ptr(), nip.data_ptr(), nix.data_ptr(), None, None)
        assert rc == _lib.ERR_INVALID and b"nnz" in lib.agcn_last_error()
    torch.cuda.synchronize()


def test_row_pointers_at_any_alignment():
    # the degree pass reads four row pointers per 16-byte load where the caller's array allows it and
    # one at a time where it does not: the same matrix through pointers at offsets 0..3 words
    import torch
    from accelgcn import degree_sort, synth
    dev = require_cuda()
    g = synth.make_config(1, "cpu", 0.5)
    want = oracle.degree_sort(g.indptr.numpy(), g.indices.numpy(), None, True)
    ix = g.indices.to(dev)
    for shift in range(4):
        buf = torch.zeros(g.n + 1 + shift, dtype=torch.int32, device=dev)
        buf[shift:] = g.indptr.to(dev)
        view = buf[shift:]
        assert view.data_ptr() % 16 == (4 * shift) % 16
        perm, nip, nix, _ = degree_sort.degree_sort_device(view, ix, None, relabel_cols=True)
        assert np.array_equal(perm.cpu().numpy(), want[0]), shift
        assert np.array_equal(nip.cpu().numpy(), want[1]) and np.array_equal(nix.cpu().numpy(), want[2]), shift


@pytest.mark.parametrize("relabel", [False, True])
@pytest.mark.parametrize("n,top", [(1, 5), (2047, 300), (2048, 3), (4095, 255), (4096, 256), (4097, 70_000), (8192, 300), (12_289, 700),
                                   (65_536, 300), (65_537, 256), (69_632, 70_000), (70_001, 17_000_000)])
def test_tile_edges_and_number_of_passes(n, top, relabel):
    # rows around the cluster's 8192 per item and its end (65 536), the sort tile (4096) and the row-pointer tile (2048) above; the largest degree decides how many of the
    # four passes move anything (255 | 256, 65 536, 2^24), and puts rows across many tiles of the permute (2048 nonzeros)
    from accelgcn import degree_sort
    require_cuda()
    rng = np.random.default_rng(n)
    deg = rng.integers(0, min(top, 60) + 1, n)
    deg[rng.integers(0, n)] = top
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    idx = rng.integers(0, n, int(indptr[-1]), dtype=np.int32)
    val = rng.random(len(idx), dtype=np.float32)
    got = degree_sort.degree_sort(indptr, idx, val, relabel_cols=relabel)
    want = oracle.degree_sort(indptr, idx, val, relabel_cols=relabel)
    for a, b, what in zip(got, want, ("perm", "indptr", "indices", "vals")):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("items", [1, 2, 3, 4, 5, 8])
def test_rows_per_thread_of_the_cluster_sort(items):
    # the cluster's shared memory is sized by the rows per thread (above three of them it needs more than the default)
    from accelgcn import degree_sort
    require_cuda()
    for n in (8192 * (items - 1) + 1, 8192 * items):
        rng = np.random.default_rng(n)
        deg = rng.integers(0, 5, n)
        deg[rng.integers(0, n, 20)] = rng.integers(250, 3_000, 20)
        indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
        idx = rng.integers(0, n, int(indptr[-1]), dtype=np.int32)
        got = degree_sort.degree_sort(indptr, idx, None, relabel_cols=True)
        for a, b, what in zip(got, oracle.degree_sort(indptr, idx, None, relabel_cols=True), ("perm", "indptr", "indices")):
            assert np.array_equal(a, b), (n, what)


@pytest.mark.parametrize("n", [3, 40, 8_192, 20_000])
@pytest.mark.parametrize("long", [2 * 256, 64 * 256, 64 * 256 + 1, 65 * 256, 96 * 256, 97 * 256 + 7, 3_000_000])
def test_rows_that_begin_many_tiles_of_the_permute(n, long):
    # the cluster sort marks where every 256th nonzero belongs: rows of up to 64 such places by their thread, longer ones
    # by the warp, one or several of them side by side, before and behind each other
    from accelgcn import degree_sort
    require_cuda()
    rng = np.random.default_rng(n + long)
    deg = rng.integers(0, 300, n)
    deg[rng.permutation(n)[:1 + min(n, 40) // 8]] = long
    deg[n // 2] = long + 1
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    idx = rng.integers(0, n, int(indptr[-1]), dtype=np.int32)
    val = rng.standard_normal(len(idx)).astype(np.float32)
    got = degree_sort.degree_sort(indptr, idx, val, relabel_cols=True)
    for a, b, what in zip(got, oracle.degree_sort(indptr, idx, val, relabel_cols=True), ("perm", "indptr", "indices", "vals")):
        assert np.array_equal(a, b), what


@pytest.mark.parametrize("n", [65_536 + 1, 65_536 * 2, 2_097_152, 2_101_249, 4_300_000])
@pytest.mark.parametrize("kind", ["low", "high", "mixed"])
def test_counters_of_tiles_groups_and_groups_of_groups(n, kind):
    # a tile of 4096 rows adds up counters of tiles, of groups of 16 and of 512 of them: sizes around their edges, with all
    # second digits zero (not counted), none zero, and some
    from accelgcn import degree_sort
    require_cuda()
    rng = np.random.default_rng(n)
    deg = rng.integers(0, 3, n)
    if kind == "high":
        deg = 256 + rng.integers(0, 200, n) if n < 200_000 else 256 * rng.integers(1, 3, n)
    if kind == "mixed":
        some = rng.random(n) < 0.05
        deg[some] = rng.integers(0, 2_000, int(some.sum()))
    indptr = np.concatenate([[0], np.cumsum(deg)])
    assert indptr[-1] < 2**31
    indptr = indptr.astype(np.int32)
    if kind == "high":                                   # the order alone: a perm for row pointers without the matrix
        import torch
        from accelgcn import _lib
        dev = torch.device("cuda")
        t, perm, nip = torch.from_numpy(indptr).to(dev), torch.empty(n, dtype=torch.int32, device=dev), torch.empty(n + 1, dtype=torch.int32, device=dev)
        _lib.check(_lib.load().agcn_degree_sort_device(t.data_ptr(), None, None, n, 0, 0, perm.data_ptr(), nip.data_ptr(), None, None, None))
        perm, nip = perm.cpu().numpy(), nip.cpu().numpy()
    else:
        idx = rng.integers(0, n, int(indptr[-1]), dtype=np.int32)
        perm, nip, nix, _ = degree_sort.degree_sort(indptr, idx, None, relabel_cols=True)
    want = np.argsort(deg, kind="stable")
    assert np.array_equal(perm, want)
    assert np.array_equal(nip, np.concatenate([[0], np.cumsum(deg[want])]))
    if kind != "high":
        inv = np.empty(n, dtype=np.int32); inv[want] = np.arange(n, dtype=np.int32)
        start = np.repeat(indptr[want] - nip[:-1], deg[want])
        assert np.array_equal(nix, inv[idx[start + np.arange(len(idx))]])


def test_release_scratch_gives_the_pool_back():
    # between calls the library keeps scratch that no other allocator of the process can use
    import torch
    import accelgcn
    from accelgcn import degree_sort
    dev = require_cuda()
    n = 4_000_000                                     # about 0.1 GB of scratch
    indptr = torch.arange(0, 2 * (n + 1), 2, dtype=torch.int32, device=dev)
    idx = torch.zeros(2 * n, dtype=torch.int32, device=dev)
    keep = degree_sort.degree_sort_device(indptr, idx, None, relabel_cols=True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(dev)[0]
    accelgcn.release_scratch()
    assert torch.cuda.mem_get_info(dev)[0] >= before + 8 * n
    again = degree_sort.degree_sort_device(indptr, idx, None, relabel_cols=True)      # and takes new scratch when it needs some
    assert all(torch.equal(a, b) for a, b in zip(keep[:3], again[:3]))


@pytest.mark.parametrize("n", [50_000, 200_000])
def test_two_graphs_in_turn_in_the_same_scratch(n):
    # the permute is resident while the kernel before it writes the new names it looks up, into the memory in which
    # the last call had other names
    import torch
    from accelgcn import degree_sort
    dev = require_cuda()
    graphs, want = [], []
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        indptr = np.concatenate([[0], np.cumsum(rng.integers(0, 12, n))]).astype(np.int32)
        idx = rng.integers(0, n, int(indptr[-1]), dtype=np.int32)
        graphs.append([torch.from_numpy(a).to(dev) for a in (indptr, idx)])
        want.append(oracle.degree_sort(indptr, idx, None, relabel_cols=True))
    for k in range(12):
        got = degree_sort.degree_sort_device(*graphs[k % 2], None, relabel_cols=True)
        for a, b in zip(got[:3], want[k % 2][:3]):
            assert np.array_equal(a.cpu().numpy(), b)
