"""Parity of the GPU SpMM with the oracle (CSR x dense in fp64, and the thread-for-thread fp32
restatement of the reference kernel), through the C ABI.  Tolerance: rel 1e-4 / abs 1e-5."""
import os

import numpy as np
import pytest

from conftest import require_cuda, spmm_close, row_abs_scale
from oracle import oracle

pytestmark = pytest.mark.gpu


class Case:
    """A degree-ordered synthetic graph on host and device with its .block4 metadata."""

    def __init__(self, cfg, scale, sort=True, empty_rows=()):
        import torch
        from accelgcn import synth, degree_sort, partition
        self.dev = require_cuda()
        g = synth.make_config(cfg, "cpu", scale)
        ip, ix, v = g.indptr.numpy(), g.indices.numpy(), g.vals.numpy()
        if len(empty_rows):                       # drop every nonzero of the named rows
            deg = np.diff(ip.astype(np.int64))
            keep = np.ones(len(ix), dtype=bool)
            for r in empty_rows:
                keep[ip[r]:ip[r + 1]] = False
                deg[r] = 0
            ix, v = ix[keep], v[keep]
            ip = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
        if sort:
            _, ip, ix, v = degree_sort.degree_sort(ip, ix, v, relabel_cols=True)
        self.n, self.indptr, self.idx, self.val = g.n, ip, ix, v
        self.block4 = partition.block_level_partition(ip)
        self.seed = g.info["seed"]
        self.t = {k: torch.from_numpy(a).to(self.dev) for k, a in
                  (("block4", self.block4), ("idx", ix), ("val", v))}

    def x(self, dim):
        from accelgcn import synth
        return synth.features(self.n, dim, self.seed, "cpu").numpy()

    def run(self, x, prefill=float("nan")):
        import torch
        from accelgcn import spmm
        xt = torch.from_numpy(x).to(self.dev)
        y = torch.full((self.n, x.shape[1]), prefill, dtype=torch.float32, device=self.dev)
        spmm.spmm(self.t["block4"], self.t["idx"], self.t["val"], xt, self.n, out=y)
        return y.cpu().numpy()

    def check(self, x, y):
        ref = oracle.spmm_csr(self.indptr, self.idx, self.val, x)
        ok = spmm_close(y, ref, row_abs_scale(self.indptr, self.val, x))
        assert not np.isnan(y).any(), "some of Y was not written"
        assert ok.all(), f"{(~ok).sum()} elements out of tolerance, first at {np.argwhere(~ok)[0]}"


@pytest.fixture(scope="module")
def cfg1():
    return Case(1, 1.0)


@pytest.fixture(scope="module")
def cfg4_small():
    return Case(4, 0.04)      # 20 000 rows, one row of 8 000 nonzeros: heavy rows crossing units


@pytest.mark.parametrize("dim", list(range(16, 129, 4)) + [1, 7, 17, 33, 61, 99, 127])
def test_config1_every_dim_against_oracle(cfg1, dim):
    x = cfg1.x(dim)
    cfg1.check(x, cfg1.run(x))


@pytest.mark.parametrize("dim", [16, 32, 60, 64, 100, 128, 45])
def test_skewed_graph_heavy_rows(cfg4_small, dim):
    x = cfg4_small.x(dim)
    y = cfg4_small.run(x)
    cfg4_small.check(x, y)


def test_matches_reference_kernel_restatement_in_fp32(cfg1):
    # against the thread-for-thread fp32 model of spmm_accel.cu on a zeroed Y
    x = cfg1.x(60)
    y = cfg1.run(x)
    ref32 = oracle.spmm_block4(cfg1.block4, cfg1.idx, cfg1.val, x, cfg1.n)
    assert spmm_close(y, ref32, row_abs_scale(cfg1.indptr, cfg1.val, x)).all()


@pytest.mark.parametrize("cfg,scale,dim", [(2, 0.02, 64), (3, 0.02, 64), (5, 0.002, 128)])
def test_other_configs_scaled_down(cfg, scale, dim):
    c = Case(cfg, scale)
    x = c.x(dim)
    c.check(x, c.run(x))


def test_overwrites_output_and_is_bitwise_reproducible(cfg4_small):
    x = cfg4_small.x(64)
    a = cfg4_small.run(x, prefill=float("nan"))
    b = cfg4_small.run(x, prefill=123.0)
    c = cfg4_small.run(x, prefill=-1e30)
    assert np.array_equal(a, b) and np.array_equal(a, c)


def test_unsorted_rows_and_zero_degree_rows_anywhere():
    # .block4 of an unsorted graph (zero-degree rows in the middle and at the end)
    n = 12_000
    c = Case(3, 0.005, sort=False, empty_rows=(0, 1, 2, 77, 78, 5000, n - 2, n - 1))
    assert c.n == n and (np.diff(c.indptr) == 0).sum() >= 8 and (np.diff(np.diff(c.indptr)) < 0).any()
    for dim in (32, 60, 9):
        x = c.x(dim)
        c.check(x, c.run(x))


def test_wide_and_strided_operands(cfg1):
    import torch
    from accelgcn import spmm
    dev = cfg1.dev
    # dim > 128 is processed in 128-column panels; ld > dim exercises the row strides
    x = cfg1.x(200)
    cfg1.check(x, cfg1.run(x))
    xw = torch.from_numpy(cfg1.x(96)).to(dev)
    ybuf = torch.full((cfg1.n, 128), float("nan"), dtype=torch.float32, device=dev)
    plan = spmm.SpmmPlan(cfg1.t["block4"], cfg1.t["idx"], cfg1.n, cfg1.n)
    plan.run(cfg1.t["idx"], cfg1.t["val"], xw[:, :64], ybuf[:, 32:96], dim=64, ldx=96, ldy=128)
    torch.cuda.synchronize()
    plan.close()
    out = ybuf.cpu().numpy()
    cfg1.check(xw[:, :64].cpu().numpy().copy(), out[:, 32:96].copy())
    assert np.isnan(out[:, :32]).all() and np.isnan(out[:, 96:]).all()       # nothing outside the panel touched


def test_linearity_at_full_size_config3_shape():
    # property that needs no oracle at a size the CPU cannot check quickly: A(ax + by) = aAx + bAy
    import torch
    from accelgcn import synth, degree_sort, partition, spmm
    dev = require_cuda()
    g = synth.make_config(3, dev, 0.25)          # 600 000 rows, ~15 M nonzeros
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals, relabel_cols=True)
    b4 = partition.block_level_partition_device(ip)
    x1 = synth.features(g.n, 64, 1, dev)
    x2 = synth.features(g.n, 64, 2, dev)
    y1 = spmm.spmm(b4, ix, v, x1, g.n)
    y2 = spmm.spmm(b4, ix, v, x2, g.n)
    y3 = spmm.spmm(b4, ix, v, 0.5 * x1 - 2.0 * x2, g.n)
    assert torch.allclose(y3, 0.5 * y1 - 2.0 * y2, rtol=1e-4, atol=1e-5)
    # and a sampled-row check against the fp64 CSR product
    rows = torch.randint(0, g.n, (300,), device=dev).tolist() + [g.n - 1]
    ip_h, ix_h, v_h, x_h = ip.cpu().numpy(), ix.cpu().numpy(), v.cpu().numpy(), x1.cpu().numpy().astype(np.float64)
    y_h = y1.cpu().numpy()
    for r in rows:
        s = slice(ip_h[r], ip_h[r + 1])
        ref = (v_h[s].astype(np.float64)[:, None] * x_h[ix_h[s]]).sum(0)
        assert np.all(np.abs(y_h[r] - ref) <= 1e-5 + 1e-4 * np.abs(ref)), r


def test_host_buffer_entry_point(cfg1):
    from accelgcn import spmm
    h = spmm.HostSpmm()
    for dim in (60, 128):
        x = cfg1.x(dim)
        y = h(cfg1.block4, cfg1.idx, cfg1.val, x, cfg1.n)
        cfg1.check(x, y)
    # constructor / run split of the plug-in: the graph goes up once, every run moves X and Y only
    h.set_graph(cfg1.block4, cfg1.idx, cfg1.val, cfg1.n, cfg1.n)
    for dim in (16, 100):
        x = cfg1.x(dim)
        cfg1.check(x, h.run(x))
    h.close()
    h2 = spmm.HostSpmm()
    with pytest.raises(spmm._lib.AccelGcnError, match="no graph set"):
        h2._n_rows, h2._n_cols = cfg1.n, cfg1.n
        h2.run(cfg1.x(16))
    h2.close()


def test_plugin_class_mirrors_reference_do_test(cfg1, tmp_path):
    # SPMM_ACCEL usage as in main.cu:131,146,166: buffers of dim_max columns, .block4 read from
    # ../block_level_meta/<graph>.block4 on every do_test, vin/vout re-read per dim
    import torch
    from accelgcn import spmm, graphio
    os.makedirs(tmp_path / "block_level_meta")
    graphio.write_block4(str(tmp_path / "block_level_meta" / "g.block4"), cfg1.block4)
    dev, n, dim_max = cfg1.dev, cfg1.n, 128
    vin = torch.from_numpy(cfg1.x(dim_max)).to(dev).reshape(-1)
    vout = torch.zeros(n * dim_max, dtype=torch.float32, device=dev)
    accel = spmm.SpmmAccel("g", torch.from_numpy(cfg1.indptr).to(dev), cfg1.t["idx"], cfg1.t["val"], vin, vout,
                           n, len(cfg1.idx), dim_max, meta_dir=str(tmp_path / "block_level_meta"))
    for dim in (60, 128):
        assert accel.do_test(False, dim) == 0.0
        x = vin[: n * dim].reshape(n, dim).cpu().numpy()
        cfg1.check(x, vout[: n * dim].reshape(n, dim).cpu().numpy())
    assert accel.do_test(True, 64) > 0.0


def test_invalid_input_is_rejected_not_faulted(cfg1):
    import torch
    from accelgcn import spmm, AccelGcnError
    dev = cfg1.dev
    bad_idx = cfg1.t["idx"].clone()
    bad_idx[5] = cfg1.n + 3
    with pytest.raises(AccelGcnError, match="column index"):
        spmm.SpmmPlan(cfg1.t["block4"], bad_idx, cfg1.n, cfg1.n)
    bad_b4 = cfg1.t["block4"].clone()
    bad_b4[3, 2] = len(cfg1.idx)                      # loc_begin past the end
    with pytest.raises(AccelGcnError, match="nonzero range"):
        spmm.SpmmPlan(bad_b4, cfg1.t["idx"], cfg1.n, cfg1.n)
    bad_b4 = cfg1.t["block4"].clone()
    bad_b4[0, 1] = cfg1.n                             # row out of range
    with pytest.raises(AccelGcnError, match="rows"):
        spmm.SpmmPlan(bad_b4, cfg1.t["idx"], cfg1.n, cfg1.n)
    torch.cuda.synchronize()


@pytest.mark.skipif(not oracle.ref_available(), reason="oracle/_ref not built (needs the reference tree at build time)")
@pytest.mark.parametrize("dim", [16, 60, 64, 100, 128])
def test_parity_with_the_reference_kernel_itself(cfg1, dim):
    # the reference's spmm_kernel_accel, compiled from its own sources for sm_100a, on a zeroed Y
    x = cfg1.x(dim)
    ref = oracle.ref_accel_spmm(cfg1.block4, cfg1.indptr, cfg1.idx, cfg1.val, x)
    y = cfg1.run(x)
    assert spmm_close(y, ref, row_abs_scale(cfg1.indptr, cfg1.val, x)).all()
    # the C restatement of that kernel is pinned by the same run
    model = oracle.spmm_block4(cfg1.block4, cfg1.idx, cfg1.val, x, cfg1.n)
    assert spmm_close(model, ref, row_abs_scale(cfg1.indptr, cfg1.val, x)).all()


@pytest.mark.skipif(not oracle.ref_available(), reason="oracle/_ref not built")
def test_parity_with_the_reference_kernel_heavy_rows(cfg4_small):
    x = cfg4_small.x(64)
    ref = oracle.ref_accel_spmm(cfg4_small.block4, cfg4_small.indptr, cfg4_small.idx, cfg4_small.val, x)
    y = cfg4_small.run(x)
    assert spmm_close(y, ref, row_abs_scale(cfg4_small.indptr, cfg4_small.val, x)).all()
    cs = oracle.ref_cusparse_spmm(cfg4_small.indptr, cfg4_small.idx, cfg4_small.val, x)
    assert spmm_close(y, cs, row_abs_scale(cfg4_small.indptr, cfg4_small.val, x)).all()


@pytest.mark.parametrize("world,slices,ranges", [(2, 1, 1), (5, 1, 1), (4, 3, 1), (8, 2, 1), (4, 1, 3), (1, 1, 2)])
def test_row_sharded_product_on_one_gpu_equals_unsharded(cfg4_small, world, slices, ranges):
    # every rank's block built and multiplied in this one process (contexts without a communicator:
    # the all-gather is replaced by assembling the gathered operand by hand): two row ranges per
    # rank, column ids renamed to gathered positions, block-local .block4
    import torch
    from accelgcn import sharded
    c = cfg4_small
    dev = c.dev
    ip, ix, v = (torch.from_numpy(a).to(dev) for a in (c.indptr, c.idx, c.val))
    x = c.x(64)
    xt = torch.from_numpy(x).to(dev)
    # (ranges > 1: the block's columns tiled into equal ranges of the gathered operand, one exchange)
    shards = [sharded.ShardedSpmm(ip, ix, v, r, world, exchange_slices=slices, communicator=False, column_ranges=ranges)
              for r in range(world)]
    gathered = shards[0].assemble_gathered([sh.to_block(xt) for sh in shards])
    blocks = []
    for sh in shards:
        y = torch.full((sh.rows_per_block, 64), float("nan"), dtype=torch.float32, device=dev)
        sh.multiply_gathered(gathered, y)
        blocks.append(y)
    torch.cuda.synchronize()
    y = shards[0].from_blocks(blocks).cpu().numpy()
    c.check(x, y)
    for sh, blk in zip(shards, blocks):                        # padding rows multiply to zero
        assert torch.all(blk[sh.rows_of() < 0] == 0)
    # the device layout is the host layout (agcn_balanced_blocks), and it balances rows and nonzeros
    ranges, per = sharded.balanced_blocks(c.indptr, world)
    per = -(-per // slices) * slices
    for r, sh in enumerate(shards):
        assert sh.rows_per_block == per and np.array_equal(sh.rows_of().cpu().numpy(), sharded.block_rows(ranges, per, r))
    nnz = np.array([sh.local_nnz for sh in shards])
    assert nnz.sum() == len(c.idx) and nnz.max() - nnz.min() <= 2 * np.diff(c.indptr).max()
    for sh in shards:
        sh.close()


def test_cpp_harness_same_cli_and_output_as_the_reference(cfg1, tmp_path):
    # spmm_test <graph> <dim>, run from a build directory beside graphs/ and block_level_meta/
    # (README.md:70-73): checks against cuSPARSE, then prints the reference's timing lines
    import subprocess, importlib.util
    from conftest import PKG
    from accelgcn import graphio
    spec = importlib.util.spec_from_file_location("agcn_build", os.path.join(PKG, "build.py"))
    mod = importlib.util.module_from_spec(spec); spec.loader.exec_module(mod)
    exe = mod.build_harness()
    graphio.write_graph(str(tmp_path / "graphs"), "synth1", cfg1.indptr, cfg1.idx)
    os.makedirs(tmp_path / "block_level_meta"); os.makedirs(tmp_path / "build")
    graphio.write_block4(str(tmp_path / "block_level_meta" / "synth1.block4"), cfg1.block4)
    out = subprocess.run([exe, "synth1", "60"], cwd=tmp_path / "build", capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "validation pass!" in out.stdout and "validation fail!" not in out.stdout
    lines = [l.split() for l in out.stdout.splitlines() if l.startswith("0/0 synth1 60 ")]
    assert [l[3] for l in lines] == ["cusparse", "accel", "accel_event"] and all(float(l[4]) > 0 for l in lines)


def test_graph_without_nonzeros_gives_zeros():
    # no tuples at all: every row is zero-filled, nothing else is launched
    import torch
    from accelgcn import spmm
    dev = require_cuda()
    n = 1000
    b4 = torch.zeros((0, 4), dtype=torch.int32, device=dev)
    empty_i = torch.zeros(0, dtype=torch.int32, device=dev)
    empty_v = torch.zeros(0, dtype=torch.float32, device=dev)
    for dim in (64, 7):
        x = torch.ones((n, dim), device=dev)
        y = torch.full((n, dim), float("nan"), device=dev)
        spmm.spmm(b4, empty_i, empty_v, x, n, out=y)
        assert torch.equal(y, torch.zeros_like(y))


def test_single_heavy_row_spanning_many_units():
    # one row of 50 000 nonzeros = 131 tuples = 17 units: all of it goes through the carry path
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    rng = np.random.default_rng(8)
    n, d = 60_000, 50_000
    indptr = np.array([0, d], dtype=np.int32)
    idx = np.sort(rng.choice(n, d, replace=False)).astype(np.int32)
    val = rng.uniform(0, 1, d).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 100)).astype(np.float32)
    b4 = partition.block_level_partition(indptr)
    assert len(b4) == 131
    y = spmm.spmm(torch.from_numpy(b4).to(dev), torch.from_numpy(idx).to(dev), torch.from_numpy(val).to(dev),
                  torch.from_numpy(x).to(dev), 1).cpu().numpy()
    ref = oracle.spmm_csr(indptr, idx, val, x)
    assert spmm_close(y, ref, row_abs_scale(indptr, val, x)).all()


def test_full_size_config2_checksum_and_sampled_rows():
    # the headline workload at its full size (250 000 nodes, ~1.2e8 nonzeros): properties that need
    # no full oracle -- 1^T (A X) = (1^T A) X in fp64, a row sample against the fp64 product, and
    # bit-identical output from two runs
    import torch
    from accelgcn import synth, degree_sort, partition, spmm
    dev = require_cuda()
    g = synth.make_config(2, dev, 1.0)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals, relabel_cols=True)
    b4 = partition.block_level_partition_device(ip)
    n, dim = g.n, 64
    x = synth.features(n, dim, 1002, dev)
    plan = spmm.SpmmPlan(b4, ix, n, n)
    y1 = torch.full((n, dim), float("nan"), device=dev)
    y2 = torch.full((n, dim), 7.0, device=dev)
    plan.run(ix, v, x, y1)
    plan.run(ix, v, x, y2)
    torch.cuda.synchronize()
    plan.close()
    assert torch.equal(y1, y2)
    col_weight = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, ix.to(torch.int64), v.to(torch.float64))
    want = col_weight @ x.to(torch.float64)                      # (1^T A) X
    got = y1.to(torch.float64).sum(0)
    assert torch.allclose(got, want, rtol=1e-6, atol=1e-6 * float(col_weight.abs().sum())), (got - want).abs().max()
    ip_h = ip.cpu().numpy()
    rows = np.unique(np.concatenate([np.random.default_rng(0).integers(0, n, 200), [0, n - 1, n - 2]]))
    for r in rows:
        a, b = int(ip_h[r]), int(ip_h[r + 1])
        ref = (v[a:b].to(torch.float64)[:, None] * x[ix[a:b].to(torch.int64)].to(torch.float64)).sum(0)
        err = (y1[r].to(torch.float64) - ref).abs()
        assert bool((err <= 1e-5 + 1e-4 * ref.abs()).all()), int(r)


# ----------------------------------------------------------------------------------------
# the configurations at the sizes the benchmark numbers are quoted on
# ----------------------------------------------------------------------------------------
def _full_config_on_device(cfg):
    import torch
    from accelgcn import synth, degree_sort, partition
    dev = require_cuda()
    g = synth.make_config(cfg, dev, 1.0)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals, relabel_cols=True)
    b4 = partition.block_level_partition_device(ip)
    seed = g.info["seed"]
    n = g.n
    del g
    torch.cuda.empty_cache()
    return dev, n, seed, ip, ix, v, b4


def _checksum_and_rows(n, ip, ix, v, x, y, n_sample=200):
    """1^T (A X) = (1^T A) X in fp64, and a row sample (with the lightest and the heaviest rows)
    against the fp64 product, at the parity tolerance rel 1e-4 / abs 1e-5 scaled by the row's
    absolute sum."""
    import torch
    dev = x.device
    assert not torch.isnan(y).any()
    col_weight = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, ix.to(torch.int64), v.to(torch.float64))
    want = col_weight @ x.to(torch.float64)
    got = y.to(torch.float64).sum(0)
    assert torch.allclose(got, want, rtol=1e-6, atol=1e-6 * float(col_weight.abs().sum())), float((got - want).abs().max())
    ip_h = ip.cpu().numpy()
    rows = np.unique(np.concatenate([np.random.default_rng(0).integers(0, n, n_sample), [0, 1, n - 3, n - 2, n - 1]]))
    xmax = float(x.abs().max())
    for r in rows:
        a, b = int(ip_h[r]), int(ip_h[r + 1])
        ref = (v[a:b].to(torch.float64)[:, None] * x[ix[a:b].to(torch.int64)].to(torch.float64)).sum(0)
        scale = max(1.0, float(v[a:b].abs().sum()) * xmax)
        err = (y[r].to(torch.float64) - ref).abs()
        assert bool((err <= 1e-5 * scale + 1e-4 * ref.abs()).all()), (int(r), float(err.max()))


@pytest.fixture(scope="module")
def cfg2_full():
    return _full_config_on_device(2)


@pytest.mark.parametrize("dim", [32, 128])
def test_full_size_config2_other_widths(cfg2_full, dim):
    # dim 128 is the launch the benchmark's roofline is quoted on, and the only one where the
    # two 64-column passes are chosen automatically (X = 128 MB against a 126 MB L2)
    import torch
    from accelgcn import synth, spmm
    dev, n, seed, ip, ix, v, b4 = cfg2_full
    x = synth.features(n, dim, seed, dev)
    plan = spmm.SpmmPlan(b4, ix, n, n)
    y = torch.full((n, dim), float("nan"), device=dev)
    plan.run(ix, v, x, y)
    torch.cuda.synchronize()
    launches = plan.info()["launches_last_run"]
    plan.close()
    if dim == 128:
        assert launches >= 2            # two column passes (plus the carry kernels if any row crosses units)
    _checksum_and_rows(n, ip, ix, v, x, y)


def test_full_size_config2_column_tiled(cfg2_full):
    # the column-tiled product at dim 128 (3 ranges): same checks, and within the parity tolerance of
    # the un-tiled product element by element (only the order of the fp32 additions differs)
    import torch
    from accelgcn import synth, spmm, _lib
    dev, n, seed, ip, ix, v, b4 = cfg2_full
    x = synth.features(n, 128, seed, dev)
    k = _lib.load().agcn_spmm_tiled_suggest(n, n, int(ix.numel()), 128)
    assert 2 <= k <= 8
    tiled = spmm.TiledSpmmPlan(ip, ix, v, n, n, dim=128)
    assert tiled.info()["n_ranges"] == k and sum(tiled.info()["range_nnz"]) == int(ix.numel())
    y1 = torch.full((n, 128), float("nan"), device=dev)
    y2 = torch.full((n, 128), 3.0, device=dev)
    tiled.run(x, y1)
    tiled.run(x, y2)
    torch.cuda.synchronize()
    tiled.close()
    assert torch.equal(y1, y2)                               # bit-identical from run to run
    _checksum_and_rows(n, ip, ix, v, x, y1)
    plan = spmm.SpmmPlan(b4, ix, n, n)
    y0 = torch.empty((n, 128), device=dev)
    plan.run(ix, v, x, y0)
    torch.cuda.synchronize()
    plan.close()
    assert bool(((y1 - y0).abs() <= 1e-5 + 1e-4 * y0.abs()).all())


@pytest.mark.parametrize("panel", [32, 64])
def test_forced_column_passes_on_small_graphs(cfg1, cfg4_small, panel, monkeypatch):
    # AGCN_SPMM_PANEL (read at plan creation) forces the pass loop -- and the reuse of the carry
    # scratch between passes -- on inputs small enough for the full oracle
    monkeypatch.setenv("AGCN_SPMM_PANEL", str(panel))
    for case in (cfg1, cfg4_small):
        for dim in (128, 100, 61):
            x = case.x(dim)
            case.check(x, case.run(x))


@pytest.mark.parametrize("panel", [48, 96, 100])
@pytest.mark.parametrize("dim", [192, 256, 301])
def test_column_passes_that_do_not_divide_a_carry_slot(cfg4_small, panel, dim, monkeypatch):
    # a slot holds 128 columns of a row that crosses units, and the arrival counters follow the last slot: a pass
    # that went on past its slot left counters that are not zero, and the plan's next product a row unwritten
    import torch
    from accelgcn import spmm
    monkeypatch.setenv("AGCN_SPMM_PANEL", str(panel))
    monkeypatch.setenv("AGCN_SPMM_PIECE", "0")
    c = cfg4_small
    plan = spmm.SpmmPlan(c.t["block4"], c.t["idx"], c.n, c.n)
    assert plan.info()["n_carry"] > 0
    x = c.x(dim)
    xt = torch.from_numpy(x).to(c.dev)
    for _ in range(3):
        y = torch.full((c.n, dim), float("nan"), device=c.dev)
        plan.run(c.t["idx"], c.t["val"], xt, y)
        c.check(x, y.cpu().numpy())
    plan.close()


@pytest.mark.parametrize("piece", [0, 7, 64, 100, 192])
def test_tuples_cut_into_pieces(cfg1, cfg4_small, piece, monkeypatch):
    # AGCN_SPMM_PIECE (read at plan creation): 0 = uncut, the form of large plans (heavy rows across units, light and
    # heavy units in turn); pieces that do not divide a row, hold several rows, or make a row cross many units
    monkeypatch.setenv("AGCN_SPMM_PIECE", str(piece))
    holes = Case(1, 0.25, empty_rows=(0, 5, 1000, 1001, 1002, 4095))
    for case in (cfg1, cfg4_small, holes):
        for dim in (128, 61, 16):
            x = case.x(dim)
            case.check(x, case.run(x))


def test_full_size_config3():
    # N = 2 400 000, ~6e7 nonzeros, dim 64: the whole product against the CPU oracle (fp64 accumulation)
    import torch
    from accelgcn import synth, spmm
    dev, n, seed, ip, ix, v, b4 = _full_config_on_device(3)
    x = synth.features(n, 64, seed, dev)
    y = torch.full((n, 64), float("nan"), device=dev)
    spmm.spmm(b4, ix, v, x, n, out=y)
    oracle.use_all_host_threads()
    ip_h, ix_h, v_h, x_h = ip.cpu().numpy(), ix.cpu().numpy(), v.cpu().numpy(), x.cpu().numpy()
    ref = oracle.spmm_csr(ip_h, ix_h, v_h, x_h)
    ok = spmm_close(y.cpu().numpy(), ref, row_abs_scale(ip_h, v_h, x_h))
    assert ok.all(), f"{(~ok).sum()} elements out of tolerance, first at {np.argwhere(~ok)[0]}"


@pytest.fixture(scope="module")
def cfg4_full():
    dev, n, seed, ip, ix, v, b4 = _full_config_on_device(4)
    host = {k: t.cpu().numpy() for k, t in (("ip", ip), ("ix", ix), ("v", v), ("b4", b4))}
    return dev, n, seed, ip, ix, v, b4, host


@pytest.mark.parametrize("dim", list(range(16, 129, 4)))
def test_full_size_config4_sweep(cfg4_full, dim):
    # N = 500 000, max degree ~9e4, every width of the configuration: against the CPU oracle and
    # (where it was built) against the reference's own kernel on the same arrays
    import torch
    from accelgcn import synth, spmm
    dev, n, seed, ip, ix, v, b4, h = cfg4_full
    x = synth.features(n, dim, seed, dev)
    y = torch.full((n, dim), float("nan"), device=dev)
    spmm.spmm(b4, ix, v, x, n, out=y)
    y_h, x_h = y.cpu().numpy(), x.cpu().numpy()
    oracle.use_all_host_threads()
    scale = row_abs_scale(h["ip"], h["v"], x_h)
    ok = spmm_close(y_h, oracle.spmm_csr(h["ip"], h["ix"], h["v"], x_h), scale)
    assert ok.all(), f"{(~ok).sum()} elements out of tolerance, first at {np.argwhere(~ok)[0]}"
    if oracle.ref_available() and dim % 16 == 0:
        ref = oracle.ref_accel_spmm(h["b4"], h["ip"], h["ix"], h["v"], x_h)
        assert spmm_close(y_h, ref, scale).all()


@pytest.mark.parametrize("dim", [17, 61, 99, 127])
def test_unaligned_widths_padded_copy_equals_scalar_path(cfg4_small, dim, monkeypatch):
    # dims that are not multiples of 4: the default copies X into aligned rows and runs the 16-byte
    # path; AGCN_SPMM_PAD=0 keeps the 4-byte gathers.  Both against the oracle, and equal to each other
    # within the tolerance (the order of additions inside a row differs between the two).
    x = cfg4_small.x(dim)
    y_pad = cfg4_small.run(x)
    cfg4_small.check(x, y_pad)
    monkeypatch.setenv("AGCN_SPMM_PAD", "0")
    y_scalar = cfg4_small.run(x)
    cfg4_small.check(x, y_scalar)
    assert spmm_close(y_pad, y_scalar, row_abs_scale(cfg4_small.indptr, cfg4_small.val, x)).all()


def test_widths_and_strides_of_any_number_type(cfg1):
    # what int() takes, as the call did before it went through the native caller
    import torch
    from accelgcn import spmm
    c = cfg1
    x = torch.from_numpy(c.x(32)).to(c.dev)
    plan = spmm.SpmmPlan(c.t["block4"], c.t["idx"], c.n, c.n)
    want, y = torch.empty((c.n, 32), device=c.dev), torch.empty((c.n, 32), device=c.dev)
    plan.run(c.t["idx"], c.t["val"], x, want)
    for number in (int, float, np.int32, np.float64, torch.tensor):
        plan.run(c.t["idx"], c.t["val"], x, y.zero_(), dim=number(32), ldx=number(32), ldy=number(32))
        assert torch.equal(y, want)
    plan.close()


def test_rows_of_x_kept_in_l2_are_rows_that_are_named_often():
    # the last rows of an X many times larger than L2 go before the others only where the nonzeros name them: not in a
    # matrix with columns in any order, not below 6x L2, not where the plan has not seen the column ids
    import ctypes
    import torch
    from accelgcn import spmm, partition, _lib
    dev = require_cuda()
    lib = _lib.load()
    l2 = torch.cuda.get_device_properties(dev).L2_cache_size
    n, mean = 2_400_000, 12
    window = int(0.45 * l2 / 512)
    indptr = torch.arange(0, (n + 1) * mean, mean, dtype=torch.int32, device=dev)
    block4 = partition.block_level_partition_device(indptr)
    gen = torch.Generator(device=dev).manual_seed(1)
    anywhere = torch.randint(0, n, (n * mean,), device=dev, generator=gen, dtype=torch.int32)

    def hot(ids, width, n_cols=n, known=True):
        col, h = ctypes.c_int64(-1), ctypes.c_void_p()
        _lib.check(lib.agcn_spmm_create(ctypes.byref(h), block4.data_ptr(), block4.shape[0], ids.data_ptr() if known else None, n, n_cols,
                                        n * mean, None))
        _lib.check(lib.agcn_spmm_plan_hot_column(h, width, ctypes.byref(col)))
        _lib.check(lib.agcn_spmm_destroy(h))
        return col.value

    assert hot(anywhere, 128) == 0
    for share, want in ((0.25, False), (0.42, True), (0.9, True)):
        # by row, as sorted rows have it: the last ids of a row are the largest
        tail = torch.rand((n, mean), device=dev, generator=gen) < share
        ids = torch.where(tail, (n - window + torch.randint(0, window, (n, mean), device=dev, generator=gen)).int(), anywhere.view(n, mean))
        ids = ids.sort(dim=1).values.contiguous()
        assert (hot(ids, 128) > 0) == want, share
        if want:
            assert hot(ids, 128) == n - window and 0 < hot(ids, 100) < n - window
            assert hot(ids, 64) == 0 or n * 64 * 4 >= 6 * l2          # the threshold is in bytes of the pass
            assert hot(ids, 128, known=False) == 0
            assert hot(ids, 128, n_cols=2 ** 31 - 2) == 0             # then the last rows are others
            # five times the columns, named at their end: passes of more than 32 columns have the kernel for it
            far = torch.where(ids >= n - window, ids + 4 * n, ids)
            assert 0 < hot(far, 64, n_cols=5 * n) < 5 * n and hot(far, 32, n_cols=5 * n) == 0
            del far
        del ids, tail


def test_product_that_starts_under_the_copy_of_x_reads_the_new_x(cfg1, cfg4_small):
    # with unaligned rows the product is resident while the copy of X it reads is still being written: X changes from
    # run to run, and every run must equal, bit for bit, the product of the same X in aligned rows
    import torch
    from accelgcn import spmm
    for c in (cfg1, cfg4_small):
        plan = spmm.SpmmPlan(c.t["block4"], c.t["idx"], c.n, c.n)
        aligned = torch.zeros((c.n, 64), device=c.dev)
        y, want = torch.empty((c.n, 61), device=c.dev), torch.empty((c.n, 64), device=c.dev)
        x = torch.from_numpy(c.x(61)).to(c.dev)
        bad = torch.zeros((), dtype=torch.int64, device=c.dev)
        for _ in range(20):
            x.mul_(-1.0).add_(0.25)
            aligned[:, :61] = x
            plan.run(c.t["idx"], c.t["val"], aligned, want)
            plan.run(c.t["idx"], c.t["val"], x, y)
            bad += (y != want[:, :61]).sum()
        assert int(bad) == 0
        plan.close()


def test_first_unaligned_width_under_stream_capture(cfg4_small):
    # the aligned copy of X is made at a width's first call.  Captured in the default mode that call is refused, as any
    # allocation is; in relaxed mode its memory outlives the graph, so that products outside of it can use it too
    import ctypes
    import torch
    from accelgcn import spmm
    from accelgcn._lib import AccelGcnError
    c, dim = cfg4_small, 61
    rt = ctypes.CDLL(next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line))
    x = c.x(dim)
    xt = torch.from_numpy(x).to(c.dev)
    y = torch.empty((c.n, dim), device=c.dev)
    side = torch.cuda.Stream(c.dev)
    stream, graph, exe = ctypes.c_void_p(side.cuda_stream), ctypes.c_void_p(), ctypes.c_void_p()
    plan = spmm.SpmmPlan(c.t["block4"], c.t["idx"], c.n, c.n)
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(stream, 0) == 0                  # cudaStreamCaptureModeGlobal
    with pytest.raises(AccelGcnError):
        plan.run(c.t["idx"], c.t["val"], xt, y, stream=side)
    rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
    rt.cudaGetLastError()
    assert rt.cudaStreamBeginCapture(stream, 2) == 0                  # cudaStreamCaptureModeRelaxed
    plan.run(c.t["idx"], c.t["val"], xt, y, stream=side)
    assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(ctypes.byref(exe), graph, ctypes.c_ulonglong(0)) == 0
    plan.run(c.t["idx"], c.t["val"], xt, y)                           # the graph has not run
    c.check(x, y.cpu().numpy())
    for _ in range(2):
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(exe, stream) == 0
        side.synchronize()
        c.check(x, y.cpu().numpy())
    assert rt.cudaGraphExecDestroy(exe) == 0 and rt.cudaGraphDestroy(graph) == 0
    plan.run(c.t["idx"], c.t["val"], xt, y)
    c.check(x, y.cpu().numpy())
    plan.close()


@pytest.mark.parametrize("case_name,dim", [("cfg1", 16), ("cfg1", 60), ("cfg4_small", 64), ("cfg4_small", 128), ("cfg4_small", 61)])
def test_products_behind_work_of_any_kind(case_name, dim, request):
    # a product is launched while the operation before it still runs, whatever that is: kernels and copies that make its
    # column ids, values and X right before, products whose result it multiplies, streams that join; also captured
    import torch
    from accelgcn import spmm
    c = request.getfixturevalue(case_name)
    idx0, val0, x0 = c.t["idx"], c.t["val"], torch.from_numpy(c.x(dim)).to(c.dev)
    plan = spmm.SpmmPlan(c.t["block4"], idx0, c.n, c.n)
    idx, val, x = torch.zeros_like(idx0), torch.empty_like(val0), torch.empty_like(x0)
    y, z = torch.empty_like(x0), torch.empty_like(x0)
    side = torch.cuda.Stream(c.dev)

    def steps(between):
        x.copy_(x0); between()
        for k in range(6):
            idx.zero_(); val.fill_(float("nan")); between()
            idx.copy_(idx0); torch.mul(val0, 0.5 + 0.125 * k, out=val); between()
            plan.run(idx, val, x, y); between()
            plan.run(idx, val, y, z, relu=True); between()
            plan.run(idx, val, z, x); between()
            x.add_(x0); between()
            side.wait_stream(torch.cuda.current_stream()); between()
            plan.run(idx, val, x, y, stream=side); between()
            torch.cuda.current_stream().wait_stream(side); between()
            plan.run(idx, val, y, z); between()
            torch.nn.functional.normalize(z, dim=1, out=x); between()
        return x

    plan.run(idx0, val0, x0, y)                      # the aligned copy of X is made outside of the capture
    want = steps(torch.cuda.synchronize).clone()
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    for _ in range(10):
        assert torch.equal(steps(lambda: None), want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        steps(lambda: None)
    for _ in range(3):
        x.fill_(float("nan"))
        graph.replay()
        assert torch.equal(x, want)
    torch.cuda.synchronize()
    plan.close()


@pytest.mark.parametrize("dim", [1, 2, 3, 5, 15, 16, 17, 31, 33, 60, 61, 63, 64, 65, 97, 127, 128, 129, 150, 259])
@pytest.mark.parametrize("kind", ["few", "pieces", "hubs"])
def test_small_products_from_rows_of_any_alignment(kind, dim):
    # small products read unaligned rows of X as they are: bit for bit what the copied, aligned rows give, whatever X holds,
    # for the launches with many and with few gathers per lane, rows that cross thread blocks, rows without nonzeros
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    rng = np.random.default_rng(dim)
    n, deg = {"few": (700, lambda: rng.integers(0, 30, 700)), "pieces": (30_000, lambda: rng.integers(0, 20, 30_000)),
              "hubs": (20_000, lambda: np.concatenate([rng.integers(0, 3, 19_990), [700, 900, 1_500, 2_000, 2_500, 3_100, 4_000, 6_000, 9_000, 20_000]]))}[kind]
    deg = np.sort(deg())
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(dev)
    nnz = int(deg.sum())
    idx = torch.from_numpy(rng.integers(0, n, nnz, dtype=np.int32)).to(dev)
    val = torch.from_numpy(rng.standard_normal(nnz).astype(np.float32)).to(dev)
    plan = spmm.SpmmPlan(partition.block_level_partition_device(indptr), idx, n, n)
    wide = (dim + 3) // 4 * 4
    xs = torch.from_numpy(rng.standard_normal((n, dim)).astype(np.float32)).to(dev)
    xs[5, 0], xs[6, dim - 1], xs[7, dim // 2] = float("inf"), float("-inf"), float("nan")
    for relu in (False, True):
        aligned, want = torch.zeros((n, wide), device=dev), torch.full((n, wide), 7.0, device=dev)
        aligned[:, :dim] = xs
        plan.run(idx, val, aligned, want, relu=relu)
        for shift, ldx, ldy in ((0, dim, dim), (1, dim, dim + 1), (3, dim + 2, wide), (2, wide + 1, dim)):
            x = torch.full((n * ldx + shift,), float("nan"), device=dev)[shift:]
            y = torch.full((n * ldy + shift,), 7.0, device=dev)[shift:]
            x.view(n, ldx)[:, :dim] = xs
            plan.run(idx, val, x, y, dim=dim, ldx=ldx, ldy=ldy, relu=relu)
            assert plan.info()["launches_last_run"] == (dim + 127) // 128            # one a pass, none for a copy
            got = y.view(n, ldy)
            assert torch.equal(got[:, :dim].nan_to_num(3.0, 4.0, 5.0), want[:, :dim].nan_to_num(3.0, 4.0, 5.0)), (relu, shift, ldx, ldy)
            assert bool((got[:, dim:] == 7.0).all())
    plan.close()


@pytest.mark.parametrize("kind", ["one row", "few", "pieces", "hubs", "mostly empty", "uncut"])
def test_product_of_a_graph_that_is_used_once(kind):
    # plan and product behind one another without a wait: the bits of a kept plan's product, whatever the number of pieces,
    # rows without nonzeros (more than their thread blocks take at a time), rows that cross thread blocks, unaligned widths
    import torch
    from accelgcn import partition, spmm, AccelGcnError
    dev = require_cuda()
    rng = np.random.default_rng(len(kind))
    deg = {"one row": lambda: [5], "few": lambda: rng.integers(0, 30, 700), "pieces": lambda: rng.integers(0, 20, 30_000),
           "hubs": lambda: np.concatenate([rng.integers(0, 3, 19_990), [700, 900, 1_500, 4_000, 6_000, 9_000, 20_000]]),
           "mostly empty": lambda: np.concatenate([np.zeros(300_000, int), rng.integers(1, 9, 2_000)]), "uncut": lambda: rng.integers(1, 5, 160_000)}[kind]()
    indptr = np.concatenate([[0], np.cumsum(np.sort(deg))]).astype(np.int32)
    n, cols, nnz = len(deg), 5_000, int(indptr[-1])
    idx = torch.from_numpy(rng.integers(0, cols, nnz, dtype=np.int32)).to(dev)
    val = torch.from_numpy(rng.standard_normal(nnz).astype(np.float32)).to(dev)
    block4 = partition.block_level_partition_device(torch.from_numpy(indptr).to(dev))
    plan = spmm.SpmmPlan(block4, idx, n, cols)
    for dim in (1, 16, 61, 64, 100, 128, 150):
        x = torch.from_numpy(rng.standard_normal((cols, dim)).astype(np.float32)).to(dev)
        want, got = torch.full((n, dim), 7.0, device=dev), torch.full((n, dim), 8.0, device=dev)
        plan.run(idx, val, x, want)
        for _ in range(3):
            assert spmm.spmm(block4, idx, val, x, n, out=got.fill_(8.0)) is got
            assert torch.equal(got, want), dim
    plan.close()
    # refused as by a plan, Y as it was; and the next product is right again
    for bad in (cols, -1):
        was, idx[nnz // 2] = int(idx[nnz // 2]), bad
        with pytest.raises(AccelGcnError, match="column index"):
            spmm.spmm(block4, idx, val, x, n, out=got.fill_(9.0))
        assert bool((got == 9.0).all())
        idx[nnz // 2] = was
    wrong = block4.clone()
    wrong[-1, 1] = n
    with pytest.raises(AccelGcnError, match="rows out of range"):
        spmm.spmm(wrong, idx, val, x, n, out=got)
    assert bool((got == 9.0).all())
    assert torch.equal(spmm.spmm(block4, idx, val, x, n, out=got), want)


@pytest.mark.parametrize("rows", [3_000, 160_000])
def test_a_graph_that_is_used_once_waits_for_its_own_stream_only(rows):
    # cut and uncut plans: Y is there when the call returns, while another stream is still busy
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    rng = np.random.default_rng(rows)
    indptr = np.concatenate([[0], np.cumsum(np.sort(rng.integers(1, 5, rows)))]).astype(np.int32)
    idx = torch.from_numpy(rng.integers(0, 500, int(indptr[-1]), dtype=np.int32)).to(dev)
    val, x = torch.rand(len(idx), device=dev), torch.rand(500, 61, device=dev)
    block4 = partition.block_level_partition_device(torch.from_numpy(indptr).to(dev))
    want, got = (torch.full((rows, 61), 7.0, device=dev) for _ in range(2))
    spmm.spmm(block4, idx, val, x, rows, out=want)
    host = torch.empty((rows, 61), pin_memory=True)
    busy, mine, done = torch.cuda.Stream(dev), torch.cuda.Stream(dev), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(2_000_000_000)            # a second or so
        done.record()
    with torch.cuda.stream(mine):
        spmm.spmm(block4, idx, val, x, rows, out=got)
        assert mine.query() and not done.query()
        host.copy_(got, non_blocking=True)
        mine.synchronize()
    assert not done.query()
    torch.cuda.synchronize()
    assert torch.equal(host, want.cpu())


def _once_graph(deg, cols, seed, dev):
    # a graph in degree order with its operands, and what a kept plan gives for it
    import torch
    from accelgcn import partition, spmm
    rng = np.random.default_rng(seed)
    indptr = np.concatenate([[0], np.cumsum(np.sort(deg))]).astype(np.int32)
    n, nnz = len(deg), int(indptr[-1])
    idx = torch.from_numpy(rng.integers(0, cols, nnz, dtype=np.int32)).to(dev)
    val = torch.from_numpy(rng.standard_normal(nnz).astype(np.float32)).to(dev)
    x = torch.from_numpy(rng.standard_normal((cols, 61 if seed % 2 else 64)).astype(np.float32)).to(dev)
    block4 = partition.block_level_partition_device(torch.from_numpy(indptr).to(dev))
    want = torch.full((n, x.shape[1]), 7.0, device=dev)
    plan = spmm.SpmmPlan(block4, idx, n, cols)
    plan.run(idx, val, x, want)
    torch.cuda.synchronize()
    plan.close()
    return block4, idx, val, x, want


def test_graphs_that_are_used_once_in_turn_in_the_same_memory():
    # the product is resident while the plan's kernel writes the tuples and carry slots that it reads, into the memory in which the
    # last graph had other ones: every row one further on, or other degrees altogether; rows that cross thread blocks in all of them
    import torch
    from accelgcn import spmm
    dev = require_cuda()
    rng = np.random.default_rng(3)
    hubs = [700, 2_000, 5_000, 9_000]
    deg = np.concatenate([rng.integers(1, 20, 9_000), hubs])
    graphs = [_once_graph(np.append(deg, [0] * zeros), 4_000, 10 + zeros, dev) for zeros in (0, 1, 2)]
    graphs += [_once_graph(np.concatenate([rng.integers(0, 20, 9_000), hubs[::2]]), 4_000, 21, dev)]
    for k in range(80):
        block4, idx, val, x, want = graphs[k % len(graphs)]
        y = spmm.spmm(block4, idx, val, x, len(want), out=torch.full_like(want, 8.0))
        assert torch.equal(y, want), k


def test_many_graphs_that_are_used_once_at_the_same_time():
    # 70 calls under way together, six more than there are words that say "something is wrong" (those are products of a plan made first): each
    # on a stream of its own that is kept busy until all have been started.  Every seventh names a column that is not there
    import threading
    import torch
    from accelgcn import spmm, AccelGcnError
    dev = require_cuda()
    rng = np.random.default_rng(4)
    graphs = [_once_graph(np.concatenate([rng.integers(0, 20, 500 + 37 * k), [900 + 10 * k]]), 1_000, k, dev) for k in range(70)]
    for k in range(0, 70, 7):
        graphs[k][1][k] = 1_000
    outs = [torch.empty_like(g[4]) for g in graphs]
    streams = [torch.cuda.Stream(dev) for _ in graphs]
    said = [None] * len(graphs)

    def one(k):
        block4, idx, val, x, want = graphs[k]
        try:
            with torch.cuda.stream(streams[k]):
                spmm.spmm(block4, idx, val, x, len(want), out=outs[k])
            said[k] = ""
        except AccelGcnError as e:
            said[k] = str(e)

    for _ in range(2):
        for o in outs:
            o.fill_(8.0)
        torch.cuda.synchronize()
        for s in streams:
            with torch.cuda.stream(s):
                torch.cuda._sleep(100_000_000)
        threads = [threading.Thread(target=one, args=(k,)) for k in range(len(graphs))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k, g in enumerate(graphs):
            if k % 7 == 0:
                assert "column index" in said[k] and bool((outs[k] == 8.0).all()), k
            else:
                assert said[k] == "" and torch.equal(outs[k], g[4]), k


@pytest.mark.parametrize("hub", [0, 3_000, 6_000])
@pytest.mark.parametrize("units", [394, 395, 444, 445, 592, 593, 932, 933])
def test_products_of_few_thread_blocks(units, hub, monkeypatch):
    # both sides of the lines between the forms of launches of few thread blocks, on graphs with and without a hub row; every slot width
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    if torch.cuda.get_device_properties(dev).multi_processor_count != 148:
        pytest.skip("sizes are those of 148 SMs")
    monkeypatch.setenv("AGCN_SPMM_PIECE", "64")
    rng = np.random.default_rng(units)
    # tuples of 12 rows of 16: three pieces; a unit is eight pieces, the hub row 47 or 94 of them
    pieces = units * 8 - (-(-hub // 64) if hub else 0)
    deg = np.full(pieces // 3 * 12 + pieces % 3 * 4, 16)
    deg = np.append(deg, hub) if hub else deg
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    n, cols = len(deg), 4_000
    idx = rng.integers(0, cols, int(indptr[-1]), dtype=np.int32)
    val = rng.standard_normal(len(idx)).astype(np.float32)
    d_idx, d_val = torch.from_numpy(idx).to(dev), torch.from_numpy(val).to(dev)
    plan = spmm.SpmmPlan(partition.block_level_partition_device(torch.from_numpy(indptr).to(dev)), d_idx, n, cols)
    assert plan.info()["n_units"] == units
    for dim in (16, 20, 32, 64, 100, 128):
        x = rng.standard_normal((cols, dim)).astype(np.float32)
        y = torch.full((n, dim), float("nan"), device=dev)
        plan.run(d_idx, d_val, torch.from_numpy(x).to(dev), y)
        assert spmm_close(y.cpu().numpy(), oracle.spmm_csr(indptr, idx, val, x), row_abs_scale(indptr, val, x)).all(), dim
    plan.close()


@pytest.fixture(scope="module", params=["many", "dense", "few"])
def uncut(request):
    # graphs whose tuples are not cut: more than 20 thread blocks per SM of light rows, of full tuples, and fewer
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    rng = np.random.default_rng(5)
    deg = {"many": lambda: np.concatenate([rng.integers(0, 4, 290_000), rng.integers(33, 90, 500), [400, 3_000, 20_000]]),
           "dense": lambda: np.concatenate([rng.integers(380, 385, 23_800), [500, 5_000]]),
           "few": lambda: np.concatenate([rng.integers(0, 5, 150_000), rng.integers(33, 200, 300), [385, 900, 7_000]])}[request.param]()
    deg = np.sort(deg)
    n, cols = len(deg), 30_000
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    idx = rng.integers(0, cols, int(indptr[-1]), dtype=np.int32)
    val = rng.standard_normal(len(idx)).astype(np.float32)
    d_idx, d_val = torch.from_numpy(idx).to(dev), torch.from_numpy(val).to(dev)
    plan = spmm.SpmmPlan(partition.block_level_partition_device(torch.from_numpy(indptr).to(dev)), d_idx, n, cols)
    yield dict(dev=dev, n=n, cols=cols, indptr=indptr, idx=idx, val=val, d_idx=d_idx, d_val=d_val, plan=plan)
    plan.close()


@pytest.mark.parametrize("dim", [33, 40, 48, 49, 56, 65, 68, 72, 81, 88, 89, 96, 104, 127, 128, 136])
def test_rows_of_x_32_bytes_at_a_time(uncut, dim):
    # uncut plans load whole eights of columns where rows of X allow it: all layouts of X and Y that do and do not, widths on
    # both sides of the rule's lines, the copy of an unaligned X in rows of eights, rows that cross thread blocks, rows without
    # nonzeros; an infinity and a NaN stay in their column
    import torch
    g = uncut
    n, cols, eights = g["n"], g["cols"], (dim + 7) // 8 * 8
    xs = np.random.default_rng(dim).standard_normal((cols, dim)).astype(np.float32)
    ref = oracle.spmm_csr(g["indptr"], g["idx"], g["val"], xs)
    scale = row_abs_scale(g["indptr"], g["val"], xs)
    touched = np.unique(np.repeat(np.arange(n), np.diff(g["indptr"]))[(g["idx"] == 7) | (g["idx"] == 9)])
    for shift, ldx, ldy, relu in ((0, dim, dim, False), (8, eights, eights, True), (4, eights, eights + 4, False), (0, eights + 4, eights, True), (1, dim, dim + 1, False)):
        x = torch.full((cols * ldx + shift,), float("nan"), device=g["dev"])[shift:]
        y = torch.full((n * ldy + shift,), 7.0, device=g["dev"])[shift:]
        x.view(cols, ldx)[:, :dim] = torch.from_numpy(xs).to(g["dev"])
        g["plan"].run(g["d_idx"], g["d_val"], x, y, dim=dim, ldx=ldx, ldy=ldy, relu=relu)
        got = y.view(n, ldy).cpu().numpy()
        assert spmm_close(got[:, :dim], np.maximum(ref, 0) if relu else ref, scale).all(), (shift, ldx, ldy)
        assert (got[:, dim:] == 7.0).all()
        x.view(cols, ldx)[7, dim - 1], x.view(cols, ldx)[9, 0] = float("inf"), float("nan")
        g["plan"].run(g["d_idx"], g["d_val"], x, y, dim=dim, ldx=ldx, ldy=ldy)
        odd = ~torch.isfinite(y.view(n, ldy)).cpu().numpy()
        assert not odd[:, 1:dim - 1].any() and not odd[:, dim:].any()
        assert np.array_equal(np.flatnonzero(odd.any(axis=1)), touched)


@pytest.mark.parametrize("dim", [40, 48, 64, 72, 88, 96, 128])
def test_bits_by_where_rows_of_x_begin(uncut, dim):
    # rows of X on 32-byte boundaries, and unaligned ones that are copied onto such, give one result whatever their stride; rows on
    # other 16-byte boundaries give one, too; rows of up to 32 nonzeros are the same in both
    import torch
    g = uncut
    n, cols = g["n"], g["cols"]
    xs = torch.from_numpy(np.random.default_rng(dim).standard_normal((cols, dim)).astype(np.float32)).to(g["dev"])

    def product(shift, ldx):
        x = torch.full((cols * ldx + shift,), float("nan"), device=g["dev"])[shift:]
        x.view(cols, ldx)[:, :dim] = xs
        y = torch.empty((n, dim), device=g["dev"])
        g["plan"].run(g["d_idx"], g["d_val"], x, y, dim=dim, ldx=ldx, ldy=dim)
        return y

    eights, quads = product(0, dim), product(4, dim)
    for shift, ldx in ((8, dim), (0, dim + 8), (1, dim), (2, dim + 1)):
        assert torch.equal(product(shift, ldx), eights), (shift, ldx)
    for shift, ldx in ((0, dim + 4), (12, dim), (4, dim + 8)):
        assert torch.equal(product(shift, ldx), quads), (shift, ldx)
    short = torch.from_numpy(np.diff(g["indptr"]) <= 32).to(g["dev"])
    assert torch.equal(eights[short], quads[short])


@pytest.mark.parametrize("dim", [33, 36, 61, 99, 123])
def test_large_products_of_an_x_that_is_named_a_few_times(dim):
    # an X of 0.4 of L2 or more with up to eight nonzeros per row is read as it is, whatever its alignment, also by uncut plans:
    # one launch, and bit for bit what the same columns in aligned rows give; rows that cross thread blocks, rows without nonzeros.
    # (Not 127 columns: an aligned 128 of such an X goes in two passes of 64, whose additions come in another order.)
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    gen = torch.Generator(dev).manual_seed(dim)
    rng = np.random.default_rng(dim)
    deg = np.sort(np.concatenate([rng.integers(0, 6, 400_000), rng.integers(33, 300, 400), [385, 4_000, 30_000]]))
    n = len(deg)
    cols = int(0.42 * torch.cuda.get_device_properties(dev).L2_cache_size / (4 * 33)) + 7
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(dev)
    nnz = int(deg.sum())
    idx = torch.randint(0, cols, (nnz,), device=dev, generator=gen, dtype=torch.int32)
    val = torch.randn(nnz, device=dev, generator=gen)
    plan = spmm.SpmmPlan(partition.block_level_partition_device(indptr), idx, n, cols)
    wide = (dim + 3) // 4 * 4
    aligned = torch.zeros((cols, wide), device=dev)
    aligned[:, :dim] = torch.randn(cols, dim, device=dev, generator=gen)
    aligned[3, 0], aligned[5, dim - 1] = float("inf"), float("nan")
    want = torch.empty((n, wide), device=dev)
    plan.run(idx, val, aligned, want, relu=True)
    plan.run(idx, val, aligned, want)
    for shift, ldx, ldy in ((1, dim, dim), (0, dim + 1, wide), (3, wide + 2, dim + 1)):
        x = torch.full((cols * ldx + shift,), float("nan"), device=dev)[shift:]
        x.view(cols, ldx)[:, :dim] = aligned[:, :dim]
        y = torch.full((n * ldy,), 7.0, device=dev)
        for _ in range(2):                  # the arrival counters are zero again
            plan.run(idx, val, x, y, dim=dim, ldx=ldx, ldy=ldy)
            assert plan.info()["launches_last_run"] == 1
        got = y.view(n, ldy)
        assert torch.equal(got[:, :dim].nan_to_num(3.0, 4.0, 5.0), want[:, :dim].nan_to_num(3.0, 4.0, 5.0)), (shift, ldx, ldy)
        assert bool((got[:, dim:] == 7.0).all())
    # and against the definition, in 64 bits
    rows = torch.repeat_interleave(torch.arange(n, device=dev), indptr.diff().long())
    finite = aligned[:, :dim].nan_to_num(0.0, 0.0, 0.0).contiguous()
    plan.run(idx, val, finite, y, dim=dim, ldx=dim, ldy=ldy)
    ref = torch.zeros((n, dim), device=dev, dtype=torch.float64).index_add_(0, rows, val.double()[:, None] * finite.double()[idx.long()])
    scale = torch.zeros(n, device=dev, dtype=torch.float64).index_add_(0, rows, val.double().abs()) * float(finite.abs().max())
    assert spmm_close(y.view(n, ldy)[:, :dim].cpu().numpy(), ref.cpu().numpy(), scale.cpu().numpy()).all()
    plan.close()


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("nnz", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 4_099, 6_000_001])
def test_a_column_id_outside_is_found_wherever_it_is(nnz, shift):
    # ids are checked 16 bytes at a time but for the ends that are not aligned: one bad id at either end, next to them and
    # inside, of arrays that begin at any of the four places of 16 bytes; small plans, and (6e6 nonzeros, uncut) large ones
    import torch
    from accelgcn import spmm, AccelGcnError
    dev = require_cuda()
    cols = 1_000
    deg = [min(384, nnz - at) for at in range(0, nnz, 384)]
    block4 = torch.from_numpy(oracle.partition(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32))).to(dev)
    room = torch.full((nnz + 8,), -1, dtype=torch.int32, device=dev)         # what lies around them is not looked at
    idx = room[shift:shift + nnz]
    idx.copy_(torch.arange(nnz, device=dev) % cols)
    idx[-1] = cols - 1
    spmm.SpmmPlan(block4, idx, len(deg), cols).close()
    for at in sorted({k for k in (0, 1, 2, 3, 4, nnz // 2, nnz - 5, nnz - 4, nnz - 3, nnz - 2, nnz - 1) if 0 <= k < nnz}):
        was = int(idx[at])
        for bad in (cols, -1, 2**31 - 1, -2**31):
            idx[at] = bad
            with pytest.raises(AccelGcnError, match="column index"):
                spmm.SpmmPlan(block4, idx, len(deg), cols)
        idx[at] = was


@pytest.mark.parametrize("rows,degree,hub,piece", [(8_192, 8, 0, 32), (9_000, 8, 0, 32), (9_268, 8, 0, 32), (9_269, 8, 0, 64), (3_000, 10, 0, 32), (3_000, 11, 0, 64),
                                                   (3_000, 11, 64, 64), (3_000, 11, 65, 32), (10_000, 4, 0, 32), (2_500, 20, 0, 64), (2_500, 20, 79, 64), (2_500, 20, 81, 32), (2_500, 20, 700, 32),
                                                   (9_472, 20, 0, 96), (9_476, 20, 0, 64), (9_476, 20, 2_000, 96), (11_500, 20, 2_000, 96),
                                                   (4_096, 40, 0, 64), (4_096, 40, 1_000, 96), (16_384, 14, 0, 64), (16_384, 8, 0, 64), (16_384, 16, 0, 64)])
def test_pieces_of_small_plans(rows, degree, hub, piece):
    # how the plan of a small graph is cut is chosen by the number of pieces: where they leave two thread blocks (of 8) per
    # SM, 8/3 with a last row of two pieces and of four times the mean, and rows of an even graph fit a piece three times
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    if torch.cuda.get_device_properties(dev).multi_processor_count != 148:
        pytest.skip("sizes are those of 148 SMs")
    deg = np.full(rows, degree)
    if hub:
        deg[-1] = hub
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    block4 = oracle.partition(indptr)

    def pieces(most):
        n = 0
        for d, _, _, info in block4:
            r, nz = (info & 0xFFFF, d) if d <= 384 else (1, info)
            if nz <= most and d <= 384:
                each = -(-r // -(-r // (most // nz)))
                n += -(-r // each)
            else:
                n += r * -(-nz // -(-nz // -(-nz // most)))
        return n

    rng = np.random.default_rng(rows)
    idx = rng.integers(0, rows, int(indptr[-1]), dtype=np.int32)
    val = rng.standard_normal(len(idx)).astype(np.float32)
    x = rng.standard_normal((rows, 33)).astype(np.float32)
    d_idx, d_val, d_x = (torch.from_numpy(a).to(dev) for a in (idx, val, x))
    y = torch.full((rows, 33), float("nan"), device=dev)
    plan = spmm.SpmmPlan(torch.from_numpy(block4).to(dev), d_idx, rows, rows)
    assert plan.info()["n_units"] == -(-pieces(piece) // 8)
    plan.run(d_idx, d_val, d_x, y)
    assert spmm_close(y.cpu().numpy(), oracle.spmm_csr(indptr, idx, val, x), row_abs_scale(indptr, val, x)).all()
    plan.close()


def test_unaligned_rows_of_a_large_operand_get_the_passes_of_the_copy():
    # few rows, an X larger than L2: a product of 128 columns runs as two passes of 64 (other slots, another order of the
    # additions in rows of more than 32 nonzeros), also from rows that are not aligned and not copied
    import torch
    from accelgcn import partition, spmm
    dev = require_cuda()
    rng = np.random.default_rng(3)
    n, cols, dim = 1_000, 260_000, 128
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(np.sort(rng.integers(0, 300, n)))]).astype(np.int32)).to(dev)
    nnz = int(indptr[-1])
    idx = torch.from_numpy(rng.integers(0, cols, nnz, dtype=np.int32)).to(dev)
    val = torch.from_numpy(rng.standard_normal(nnz).astype(np.float32)).to(dev)
    plan = spmm.SpmmPlan(partition.block_level_partition_device(indptr), idx, n, cols)
    xs = torch.randn(cols, dim, device=dev, generator=torch.Generator(dev).manual_seed(1))
    want = torch.empty((n, dim), device=dev)
    plan.run(idx, val, xs, want)
    assert plan.info()["launches_last_run"] == 2
    for ldx, shift in ((129, 0), (128, 1), (131, 2)):
        x = torch.full((cols * ldx + shift,), float("nan"), device=dev)[shift:]
        x.view(cols, ldx)[:, :dim] = xs
        got = torch.empty((n, dim), device=dev)
        plan.run(idx, val, x, got, dim=dim, ldx=ldx, ldy=dim)
        assert plan.info()["launches_last_run"] == 2                 # no copy
        assert torch.equal(got, want), (ldx, shift)
    plan.close()


@pytest.mark.parametrize("case_name", ["cfg1", "cfg4_small"])
def test_column_tiled_small(case_name, request):
    # tiled plan with several range layouts (one of them empty), ReLU, an unaligned width and the
    # range-by-range entry, against the oracle
    import torch
    from accelgcn import spmm
    c = request.getfixturevalue(case_name)
    dev = c.dev
    ip = torch.from_numpy(c.indptr).to(dev)
    n = c.n
    for bounds in ([0, n], [0, n // 2, n], [0, n // 3, n // 3, n - 5, n]):
        tiled = spmm.TiledSpmmPlan(ip, c.t["idx"], c.t["val"], n, n, bounds=bounds)
        for dim, relu in ((64, False), (128, True), (33, True)):
            x = c.x(dim)
            xt = torch.from_numpy(x).to(dev)
            y = torch.full((n, dim), float("nan"), device=dev)
            tiled.run(xt, y, relu=relu)
            y2 = torch.full((n, dim), float("nan"), device=dev)
            for k in range(len(bounds) - 1):
                tiled.run(xt, y2, relu=relu, only_range=k)
            torch.cuda.synchronize()
            assert torch.equal(y, y2)
            ref = oracle.spmm_csr(c.indptr, c.idx, c.val, x)
            if relu:
                ref = np.maximum(ref, 0)
            assert spmm_close(y.cpu().numpy(), ref, row_abs_scale(c.indptr, c.val, x)).all(), (bounds, dim)
        tiled.close()


def test_host_batch_and_streamed_graph(cfg1, cfg4_small):
    # the pipelined host-buffer calls: several products on a resident graph, and graph + products in
    # one call (A uploaded and multiplied range by range); bit-identical to the one-product call
    import torch
    from accelgcn import spmm
    for c in (cfg1, cfg4_small):
        h = spmm.HostSpmm()
        dims = [32, 64, 128, 60, 33]
        xs = [np.ascontiguousarray(c.x(d)) for d in dims]
        ys = h.step_batch(c.block4, c.idx, c.val, xs[:4], c.n)              # streamed, in one range: these plans are cut
        for x, y in zip(xs[:4], ys):
            c.check(x, y)
        t = h.last_timing()                                                  # where the time of that call went
        assert 0 <= t["first_kernel_started"] <= t["last_kernel_finished"] <= t["last_y_downloaded"] + 1e-3
        assert t["a_uploaded"] > 0 and t["host_all_enqueued"] >= t["host_plan_built"] > 0
        ys_all = h.step_batch(c.block4, c.idx, c.val, xs, c.n)              # 33 columns: through an aligned copy of X
        for x, y in zip(xs, ys_all):
            c.check(x, y)
        h.set_graph(c.block4, c.idx, c.val, c.n, c.n)
        ys_res = h.run_batch(xs)
        for a, b in zip(ys_all, ys_res):
            assert np.array_equal(a, b)
        for x, y in zip(xs, ys_res):
            assert np.array_equal(h.run(x), y)
        for a, b in zip(ys, ys_res[:4]):
            assert np.array_equal(a, b)
        # pinned buffers take the same path
        px = [torch.from_numpy(x).pin_memory() for x in xs[:3]]
        py = [torch.empty((c.n, d), dtype=torch.float32).pin_memory() for d in dims[:3]]
        h.run_batch(px, outs=py)
        for y, ref in zip(py, ys_res[:3]):
            assert np.array_equal(y.numpy(), ref)
        # a column id out of range is rejected (by the check that runs ahead of each range), nothing faults
        bad = c.idx.copy()
        bad[len(bad) // 2] = c.n + 7
        with pytest.raises(spmm._lib.AccelGcnError, match="column index"):
            h.step_batch(c.block4, bad, c.val, xs[:3], c.n)
        ys_again = h.step_batch(c.block4, c.idx, c.val, xs[:3], c.n)        # and the context is still good
        for a, b in zip(ys_again, ys_res[:3]):
            assert np.array_equal(a, b)
        h.close()


def test_streamed_graph_in_several_ranges_and_malformed_block4():
    # a graph large enough (2.4e7 nonzeros) for the streamed call to cut A into several upload ranges:
    # bit-identical to the resident product; and tuples that would put a cut outside the arrays or out of
    # order (the cuts are taken from the caller's .block4 before the plan has validated it) are an error,
    # not a fault
    from accelgcn import spmm
    c = Case(2, 0.2)
    assert len(c.idx) * 8 >> 25 >= 4
    h = spmm.HostSpmm()
    # widths that are no multiple of 4 go through an aligned copy of X per product, made when that X has arrived; the
    # products' ranges interleave and every one keeps its own partial sums
    odd = [np.ascontiguousarray(c.x(d)) for d in (33, 64, 61)]
    want = [c.run(x) for x in odd]
    c.check(odd[2], want[2])
    for y, w in zip(h.step_batch(c.block4, c.idx, c.val, odd, c.n), want):
        assert np.array_equal(y, w)
    t = h.last_timing()                                   # of the streamed form, whatever the widths: an error after another
    assert 0 <= t["first_kernel_started"] <= t["last_kernel_finished"]
    h.set_graph(c.block4, c.idx, c.val, c.n, c.n)
    for y, w in zip(h.run_batch(odd), want):
        assert np.array_equal(y, w)
    xs = [np.ascontiguousarray(c.x(d)) for d in (32, 64)]
    ys = h.step_batch(c.block4, c.idx, c.val, xs, c.n)
    for x, y in zip(xs, ys):
        assert np.array_equal(y, c.run(x))
    n_units = (len(c.block4) + 7) // 8
    for unit, loc in ((n_units // 3, len(c.idx) + 5), (n_units // 2, 3), (2 * n_units // 3, -7)):
        bad = c.block4.copy()
        bad[unit * 8, 2] = loc
        with pytest.raises(spmm._lib.AccelGcnError):
            h.step_batch(bad, c.idx, c.val, xs, c.n)
    bad = c.block4.copy()
    bad[(n_units // 2) * 8, 1] = c.n + 1                 # row of a unit's first tuple past the matrix
    with pytest.raises(spmm._lib.AccelGcnError):
        h.step_batch(bad, c.idx, c.val, xs, c.n)
    ys_again = h.step_batch(c.block4, c.idx, c.val, xs, c.n)           # the context is still good
    for a, b in zip(ys_again, ys):
        assert np.array_equal(a, b)
    h.close()


def test_cpp_harness_full_sweep_mode(cfg1, tmp_path):
    # spmm_test with no arguments: every graph of ../graphs at every dim 16..128 step 1
    # (main.cu:195-219), here on two small graphs; with checking forced on, every product validates
    import subprocess, importlib.util
    from conftest import PKG
    from accelgcn import graphio, degree_sort, partition, synth
    spec = importlib.util.spec_from_file_location("agcn_build", os.path.join(PKG, "build.py"))
    mod = importlib.util.module_from_spec(spec); spec.loader.exec_module(mod)
    exe = mod.build_harness()
    os.makedirs(tmp_path / "block_level_meta"); os.makedirs(tmp_path / "build")
    graphio.write_graph(str(tmp_path / "graphs"), "synth1", cfg1.indptr, cfg1.idx)
    graphio.write_block4(str(tmp_path / "block_level_meta" / "synth1.block4"), cfg1.block4)
    g = synth.make_config(4, "cpu", 0.004)
    _, ip, ix, _ = degree_sort.degree_sort(g.indptr.numpy(), g.indices.numpy(), None)
    graphio.write_graph(str(tmp_path / "graphs"), "synth4", ip, ix)
    graphio.write_block4(str(tmp_path / "block_level_meta" / "synth4.block4"), partition.block_level_partition(ip))
    env = dict(os.environ, AGCN_TEST_CHECK_ALL="1")
    out = subprocess.run([exe], cwd=tmp_path / "build", capture_output=True, text=True, timeout=1200, env=env)
    assert out.returncode == 0, out.stdout[-2000:] + out.stderr[-2000:]
    assert "validation fail!" not in out.stdout
    accel = [l.split() for l in out.stdout.splitlines() if " accel " in l]
    assert len(accel) == 2 * 113 and {l[1] for l in accel} == {"synth1", "synth4"}
    assert sorted({int(l[2]) for l in accel}) == list(range(16, 129))
    assert out.stdout.count("validation pass!") == 2 * 113


def test_degree_sort_files_front_end(tmp_path):
    # original-order files -> .new_indptr / .new_indices / .perm, as one library call
    from accelgcn import graphio, synth
    g = synth.make_config(1, "cpu", 0.25)
    ip, ix = g.indptr.numpy(), g.indices.numpy()
    d = str(tmp_path / "graphs")
    graphio.write_graph(d, "g", np.zeros(1, np.int32), np.zeros(0, np.int32), orig_indptr=ip, orig_indices=ix)
    perm, nip, nix = graphio.degree_sort_files(d, "g")
    want = oracle.degree_sort(ip, ix, None, True)
    assert np.array_equal(perm, want[0]) and np.array_equal(nip, want[1]) and np.array_equal(nix, want[2])
    rip, rix = graphio.read_sorted_graph(d, "g")
    assert np.array_equal(rip, nip) and np.array_equal(rix, nix)
    assert np.array_equal(graphio.read_array(os.path.join(d, "g.perm")), perm)


def test_gather_probe_runs():
    import ctypes
    from accelgcn import _lib
    require_cuda()
    gbs = ctypes.c_double(0.0)
    _lib.check(_lib.load().agcn_probe_gather_bandwidth(1 << 16, 64, 1 << 22, 3, 5, ctypes.byref(gbs)))
    assert gbs.value > 100.0            # GB/s: any working GPU is far above this
