"""The dense transform (tcgen05 TF32 GEMM) and the two-layer GCN forward against fp64 numpy.

TF32 keeps 10 mantissa bits of each operand: with K = 128 products per output the tolerance is
rel 2e-3 of the row scale (sum_k |h_k w_kn|) -- stated here, separate from the fp32 SpMM gate."""
import numpy as np
import pytest

from conftest import require_cuda

pytestmark = pytest.mark.gpu


def _check_gemm(h, w, z):
    ref = h.astype(np.float64) @ w.astype(np.float64)
    scale = np.abs(h).astype(np.float64) @ np.abs(w).astype(np.float64)
    err = np.abs(z - ref)
    assert not np.isnan(z).any()
    assert np.all(err <= 2e-3 * scale + 1e-6), f"max err/scale {np.max(err / (scale + 1e-30)):.2e}"


@pytest.mark.parametrize("m", [1, 127, 128, 129, 1000, 128 * 148 + 5, 300_000])
def test_gemm_tf32_matches_fp64(m):
    import torch
    from accelgcn import gemm, synth
    dev = require_cuda()
    h = synth.features(m, 128, 11 + m, dev)
    w = synth.glorot(128, 128, 5, 8, dev)
    z = torch.full((m, 128), float("nan"), device=dev)
    gemm.gemm_tf32(h, w, out=z)
    torch.cuda.synchronize()
    _check_gemm(h.cpu().numpy(), w.cpu().numpy(), z.cpu().numpy())


@pytest.mark.parametrize("m", [1, 127, 128, 129, 128 * 148 + 5, 128 * 148 * 2, 128 * 148 * 5 + 77])
def test_pair_of_transforms_matches_fp64(m):
    # relu(P W1) W2 in one kernel, thread blocks with one to six tiles: their two accumulators of either product take turns.
    # P, W1 and W2 are cut to TF32 (2^-10 each), the activations rounded (2^-11); relu does not stretch an error
    import torch
    from accelgcn import gemm, synth
    dev = require_cuda()
    p = synth.features(m, 128, 17 + m, dev)
    w1, w2 = synth.glorot(128, 128, 5, 8, dev), synth.glorot(128, 128, 5, 9, dev)
    z = torch.full((m + 2, 128), float("nan"), device=dev)
    status = torch.full((1,), 9, dtype=torch.int32, device=dev)
    gemm.gemm_tf32_pair_async(p, w1, w2, z[:m], status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and bool(torch.isnan(z[m:]).all())
    p64, w1_64, w2_64 = p.double(), w1.double(), w2.double()
    h = (p64 @ w1_64).clamp_(min=0)
    bound = 2e-3 * (p64.abs() @ w1_64.abs()) @ w2_64.abs() + 1.5e-3 * h @ w2_64.abs() + 1e-6
    assert bool(((z[:m].double() - h @ w2_64).abs() <= bound).all())
    # values that TF32 holds, through the identity twice: exact
    p = torch.randint(-512, 512, (m, 128), device=dev).float() / 64.0
    eye = torch.eye(128, device=dev)
    gemm.gemm_tf32_pair_async(p, eye, eye, z[:m], status)
    assert torch.equal(z[:m], p.clamp(min=0)) and int(status.item()) == 0
    # an activation above the largest TF32 number, which the nearest one would be infinity for: cut
    p.zero_()
    w1 = eye.clone()
    w1[1, 0] = 1.0
    p[m - 1, 0], p[m - 1, 1] = float.fromhex("0x1.ffcp127"), float.fromhex("0x1.8p116")
    gemm.gemm_tf32_pair_async(p, w1, eye, z[:m], status)
    assert float(z[m - 1, 0]) == float.fromhex("0x1.ffcp127") and bool(torch.isfinite(z[:m]).all())


def test_gemm_identity_and_strided_rows():
    import torch
    from accelgcn import gemm, synth
    dev = require_cuda()
    # values exactly representable in TF32 times the identity: the product is exact
    h = torch.randint(-512, 512, (5000, 128), device=dev).to(torch.float32) / 64.0
    z = gemm.gemm_tf32(h, torch.eye(128, device=dev))
    assert torch.equal(z, h)
    # operands with a row stride larger than 128; columns outside the product are untouched
    big = synth.features(777, 256, 3, dev)
    out = torch.full((777, 192), float("nan"), device=dev)
    w = synth.glorot(128, 128, 5, 9, dev)
    gemm.gemm_tf32(big[:, 64:192], w, out=out[:, :128])
    torch.cuda.synchronize()
    _check_gemm(big[:, 64:192].cpu().numpy(), w.cpu().numpy(), out[:, :128].cpu().numpy())
    assert torch.isnan(out[:, 128:]).all()


def test_gemm_rejects_other_shapes():
    import torch
    from accelgcn import gemm, AccelGcnError
    dev = require_cuda()
    with pytest.raises(AccelGcnError, match="K = N = 128"):
        gemm.gemm_tf32(torch.zeros((10, 64), device=dev), torch.zeros((64, 128), device=dev))


def test_spmm_fused_relu():
    import torch
    from accelgcn import synth, degree_sort, partition, spmm
    from oracle import oracle
    dev = require_cuda()
    g = synth.make_config(4, dev, 0.02)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals)
    b4 = partition.block_level_partition_device(ip)
    x = synth.features(g.n, 64, 4, dev)
    plan = spmm.SpmmPlan(b4, ix, g.n, g.n)
    y = torch.full((g.n, 64), float("nan"), device=dev)
    plan.run(ix, v, x, y, relu=True)
    torch.cuda.synchronize()
    plan.close()
    ref = np.maximum(oracle.spmm_csr(ip.cpu().numpy(), ix.cpu().numpy(), v.cpu().numpy(), x.cpu().numpy()), 0)
    y = y.cpu().numpy()
    assert (y >= 0).all() and np.all(np.abs(y - ref) <= 1e-4 * np.abs(ref) + 5e-4)


def test_gemm_async_entry_and_status_word():
    import torch
    from accelgcn import gemm, synth
    dev = require_cuda()
    h = synth.features(70_000, 128, 3, dev)
    w = synth.glorot(128, 128, 5, 8, dev)
    z = torch.full((70_000, 128), float("nan"), device=dev)
    status = torch.full((1,), 77, dtype=torch.int32, device=dev)         # the call zeroes it on the stream
    gemm.gemm_tf32_async(h, w, z, status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    _check_gemm(h.cpu().numpy(), w.cpu().numpy(), z.cpu().numpy())
    assert torch.equal(z, gemm.gemm_tf32(h, w))                          # same kernel, same bits


def test_gemm_bounded_wait_runs_out_and_the_next_call_succeeds():
    # failure detection without a fault: the self-test entry starves one pipeline wait (a load that
    # is never issued) under a spin limit of well under a millisecond; the kernel must leave through
    # its abort path -- status AGCN_ERR_CUDA, tensor memory freed -- and the device must stay usable
    import torch
    from accelgcn import gemm, synth, _lib
    dev = require_cuda()
    h = synth.features(40_000, 128, 4, dev)
    w = synth.glorot(128, 128, 5, 9, dev)
    z = torch.zeros((40_000, 128), device=dev)
    rc = gemm.selftest_timeout(h, w, z)
    assert rc == _lib.ERR_CUDA and b"ran out" in _lib.load().agcn_last_error()
    torch.cuda.synchronize()                                             # no sticky error: the context is intact
    for _ in range(2):
        z2 = gemm.gemm_tf32(h, w)
        torch.cuda.synchronize()
        _check_gemm(h.cpu().numpy(), w.cpu().numpy(), z2.cpu().numpy())


@pytest.mark.parametrize("m", [1, 128 * 5, 128 * 700 + 9])
def test_bounded_wait_of_the_pair_of_transforms_runs_out_and_the_next_call_succeeds(m):
    # the same for the kernel that makes both, thread blocks with one tile and with several: all its warps leave, whichever of
    # them gives up first
    import torch
    from accelgcn import gemm, synth, _lib
    dev = require_cuda()
    p, z = synth.features(m, 128, 4, dev), torch.zeros((m, 128), device=dev)
    w1, w2 = (synth.glorot(128, 128, 5, k, dev) for k in (8, 9))
    status = torch.full((1,), 9, dtype=torch.int32, device=dev)
    want = torch.empty_like(z)
    gemm.gemm_tf32_pair_async(p, w1, w2, want, status)
    for _ in range(5):
        assert gemm.pair_selftest_timeout(p, w1, w2, z) == _lib.ERR_CUDA and b"ran out" in _lib.load().agcn_last_error()
        gemm.gemm_tf32_pair_async(p, w1, w2, z, status)
        torch.cuda.synchronize()
        assert int(status.item()) == 0 and torch.equal(z, want)


@pytest.mark.parametrize("m", [1, 128 * 5, 128 * 300])
def test_gemm_error_of_any_thread_block_is_reported_every_time(m):
    # the status word is zeroed on the stream and not by a thread block of the launch that may report into it
    import torch
    from accelgcn import gemm, synth, _lib
    dev = require_cuda()
    h, w = synth.features(m, 128, 4, dev), synth.glorot(128, 128, 5, 9, dev)
    z = torch.zeros((m, 128), device=dev)
    for _ in range(10):
        assert gemm.selftest_timeout(h, w, z) == _lib.ERR_CUDA
    want = gemm.gemm_tf32(h, w)
    status = torch.full((1,), 5, dtype=torch.int32, device=dev)          # what an earlier launch left is gone too
    gemm.gemm_tf32_async(h, w, z, status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and torch.equal(z, want)


def test_forward_times_of_the_last_of_several_runs():
    # the transforms note their own begin and end; the end only grows and is never cleared by a run
    import torch
    from accelgcn import synth, degree_sort, sharded, gcn
    dev = require_cuda()
    g = synth.make_config(5, dev, 0.0005)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals)
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    fwd = gcn.GcnForward(sh, [synth.glorot(128, 128, 1005, k, dev) for k in (8, 9)])
    x = sh.to_block(synth.features(g.n, 128, 1005, dev))
    for runs in (1, 3, 2):
        for _ in range(runs):
            fwd.forward(x)
        torch.cuda.synchronize()
        times = fwd.status(timings=True)
        # one run of 25 000 nodes is well below a millisecond; times that span several runs or none are not
        assert all(t >= 0 for layer in times for t in layer) and all(layer[0] > 0 and layer[2] > 0 for layer in times)
        assert sum(t for layer in times for t in layer) < 5.0
    fwd.close(); sh.close()


def _forward_reference(ip_h, ix_h, v_h, x_h, w1_h, w2_h):
    """CPU forward: fp32 storage, dense transform in fp64 row blocks, SpMM with fp64 accumulation (oracle)."""
    from oracle import oracle
    oracle.use_all_host_threads()

    def dense(h, w):
        out = np.empty((h.shape[0], w.shape[1]), dtype=np.float32)
        w64 = w.astype(np.float64)
        for a in range(0, h.shape[0], 1 << 18):
            out[a:a + (1 << 18)] = h[a:a + (1 << 18)].astype(np.float64) @ w64
        return out

    h1 = np.maximum(oracle.spmm_csr(ip_h, ix_h, v_h, dense(x_h, w1_h)), 0)
    return np.maximum(oracle.spmm_csr(ip_h, ix_h, v_h, dense(h1, w2_h)), 0)


@pytest.mark.parametrize("world,slices", [(1, 1), (3, 1), (4, 2)])
def test_two_layer_gcn_forward_matches_fp64(world, slices):
    # config 5 scaled to 25 000 nodes; with world > 1 every rank's block runs in this process
    # (contexts without a communicator) and the all-gather is assembled by hand; the NCCL exchange
    # itself runs in the multi-GPU benchmark and its layout is covered by the gloo tests
    import torch
    from accelgcn import synth, degree_sort, sharded, gemm, gcn
    dev = require_cuda()
    g = synth.make_config(5, dev, 0.0005)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals)
    n = g.n
    x = synth.features(n, 128, 1005, dev)
    w1, w2 = synth.glorot(128, 128, 1005, 8, dev), synth.glorot(128, 128, 1005, 9, dev)
    shards = [sharded.ShardedSpmm(ip, ix, v, r, world, exchange_slices=slices, communicator=False) for r in range(world)]

    def layer(h_blocks, w):
        zs = [gemm.gemm_tf32(hb, w) for hb in h_blocks]
        zg = shards[0].assemble_gathered(zs)
        outs = []
        for sh in shards:
            y = torch.empty((sh.rows_per_block, 128), device=dev)
            sh.multiply_gathered(zg, y, relu=True)
            outs.append(y)
        return outs

    out_blocks = layer(layer([sh.to_block(x) for sh in shards], w1), w2)
    out = shards[0].from_blocks(out_blocks).cpu().numpy()
    ref = _forward_reference(ip.cpu().numpy(), ix.cpu().numpy(), v.cpu().numpy(), x.cpu().numpy(), w1.cpu().numpy(), w2.cpu().numpy())
    scale = np.abs(ref).max()
    assert np.all(np.abs(out - ref) <= 4e-3 * scale), np.abs(out - ref).max() / scale
    if world == 1:
        # the native forward (agcn_gcn2_forward_*) enqueues the same kernels: same bits
        fwd = gcn.GcnForward(shards[0], [w1, w2])
        got = fwd.forward(shards[0].to_block(x))
        torch.cuda.synchronize()
        times = fwd.status(timings=True)
        assert len(times) == 2 and all(t >= 0 for layer_t in times for t in layer_t)
        assert torch.equal(got, out_blocks[0])
        fwd.close()
    for sh in shards:
        sh.close()


@pytest.mark.parametrize("n,launches", [(32_767, 4), (32_768, 3)])
def test_forward_on_both_sides_of_the_line(n, launches):
    # from 32 768 rows on A is applied to X before W1 and one kernel makes both transforms: the same function, TF32 in the transforms
    import torch
    from accelgcn import synth, sharded, gcn
    dev = require_cuda()
    gen = torch.Generator(dev).manual_seed(n)
    ip = torch.arange(0, 5 * n + 1, 5, dtype=torch.int32, device=dev)
    ix = torch.randint(0, n, (5 * n,), dtype=torch.int32, device=dev, generator=gen)
    v = torch.rand(5 * n, device=dev, generator=gen)
    x = synth.features(n, 128, 3, dev)
    w = [synth.glorot(128, 128, 3, k, dev) for k in (8, 9)]
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    fwd = gcn.GcnForward(sh, w)
    out = fwd.forward(sh.to_block(x))
    torch.cuda.synchronize()
    times = fwd.status(timings=True)
    assert fwd.launches() == launches and fwd.paired() == (launches == 3) and all(layer[0] > 0 and layer[2] > 0 for layer in times)

    def times_a(h):
        return (h[ix.long()] * v.double()[:, None]).view(n, 5, 128).sum(dim=1)

    ref = times_a(times_a(x.double() @ w[0].double()).clamp_(min=0) @ w[1].double()).clamp_(min=0)
    assert float((out.double() - ref).abs().max()) <= 4e-3 * float(ref.max())
    fwd.close(); sh.close()


@pytest.mark.parametrize("n,mean", [(32_768, 8), (40_000, 20), (250_000, 12)])
def test_paired_forward_is_its_three_calls_in_turn(n, mean):
    # plans that cut their tuples and plans that do not, hub rows, W written right before the forward: the bits of A X,
    # agcn_gemm_tf32_pair_async and relu(A Z) called one after the other, from run to run and with the result in place of X
    import torch
    from accelgcn import synth, sharded, gcn, gemm, degree_sort, partition, spmm
    dev = require_cuda()
    g = synth.chung_lu("powerlaw", n, synth.power_law_weights(n, 2.2, float(mean), n / 4), n * mean, 1, dev)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals, relabel_cols=True)
    x = synth.features(n, 128, 3, dev)
    w1, w2 = (synth.glorot(128, 128, 3, k, dev) for k in (8, 9))
    plan = spmm.SpmmPlan(partition.block_level_partition_device(ip), ix, n, n)
    p, z, want = (torch.full_like(x, float("nan")) for _ in range(3))
    status = torch.full((1,), 9, dtype=torch.int32, device=dev)
    plan.run(ix, v, x, p)
    gemm.gemm_tf32_pair_async(p, w1, w2, z, status)
    plan.run(ix, v, z, want, relu=True)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    plan.close()
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    late = [torch.zeros_like(w1), torch.zeros_like(w2)]
    fwd = gcn.GcnForward(sh, late)
    block = sh.to_block(x)
    for _ in range(3):
        for t, w in zip(late, (w1, w2)):
            t.fill_(float("nan"))
            t.copy_(w)
        assert torch.equal(fwd.forward(block)[:n], want) and fwd.paired()
    assert torch.equal(fwd.forward(block, out=block)[:n], want)
    fwd.status(); fwd.close(); sh.close()


def test_two_layer_gcn_forward_at_five_million_nodes():
    # configuration 5 at a tenth of its size (N = 5 000 000, ~1.07e8 nonzeros, 128 features): the whole
    # native forward against the CPU forward.  Tolerance: TF32 keeps 10 mantissa bits per operand of
    # the dense transform, so 4e-3 of the output scale (the SpMM itself is fp32 within 1e-4).
    import torch
    from accelgcn import synth, degree_sort, sharded, gcn
    dev = require_cuda()
    g = synth.make_config(5, dev, 0.1)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals)
    n = g.n
    del g
    x = synth.features(n, 128, 1005, dev)
    w1, w2 = synth.glorot(128, 128, 1005, 8, dev), synth.glorot(128, 128, 1005, 9, dev)
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    fwd = gcn.GcnForward(sh, [w1, w2])
    out_block = fwd.forward(sh.to_block(x))
    torch.cuda.synchronize()
    fwd.status()
    out = sh.from_blocks([out_block]).cpu().numpy()
    fwd.close(); sh.close()
    ref = _forward_reference(ip.cpu().numpy(), ix.cpu().numpy(), v.cpu().numpy(), x.cpu().numpy(), w1.cpu().numpy(), w2.cpu().numpy())
    scale = float(np.abs(ref).max())
    err = np.abs(out - ref)
    assert err.max() <= 4e-3 * scale, err.max() / scale
    # and tighter where it matters: the typical element, not just the worst one
    assert float(np.sqrt((err.astype(np.float64) ** 2).mean())) <= 4e-4 * scale


@pytest.mark.parametrize("m,n_cols", [(1, 64), (127, 500), (1000, 5000), (128 * 300 + 17, 40_000)])
def test_fused_layer_matches_fp64(m, n_cols):
    # Z2 = relu(A Z1) W for rows of 0..32 nonzeros: the sparse part in fp32 (rel 1e-4), the dense part in
    # TF32 (2e-3 of the row scale sum_k |h_k w_kn|)
    import torch
    from accelgcn import gemm, synth
    dev = require_cuda()
    rng = np.random.default_rng(m)
    deg = rng.integers(0, 33, m)
    deg[rng.integers(0, m, max(1, m // 50))] = 0
    deg[rng.integers(0, m, max(1, m // 50))] = 32
    ip = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    ix = rng.integers(0, n_cols, int(ip[-1])).astype(np.int32)
    v = rng.uniform(-1, 1, int(ip[-1])).astype(np.float32)
    z1 = synth.features(n_cols, 128, 77 + m, dev)
    w = synth.glorot(128, 128, 5, 9, dev)
    out = torch.full((m + 3, 128), float("nan"), device=dev)
    gemm.gcn_fused_layer(torch.from_numpy(ip).to(dev), torch.from_numpy(ix).to(dev), torch.from_numpy(v).to(dev), z1, w, m,
                         out=out[:m])
    torch.cuda.synchronize()
    assert torch.isnan(out[m:]).all()                       # rows past m_rows are not written
    z1_h, w_h = z1.cpu().numpy().astype(np.float64), w.cpu().numpy().astype(np.float64)
    h = np.zeros((m, 128))
    rows = np.repeat(np.arange(m), deg)
    np.add.at(h, rows, v[:, None].astype(np.float64) * z1_h[ix])
    h = np.maximum(h, 0)
    ref = h @ w_h
    scale = np.abs(h) @ np.abs(w_h)
    got = out[:m].cpu().numpy()
    assert not np.isnan(got).any()
    assert np.all(np.abs(got - ref) <= 2e-3 * scale + 1e-5), float(np.max(np.abs(got - ref) / (scale + 1e-30)))


def _captured_nodes(forward, x):
    """Operations one forward enqueues: kernels, memsets and event records of a captured run."""
    import ctypes
    import torch
    rt = ctypes.CDLL(next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line))
    side, graph, n = torch.cuda.Stream(), ctypes.c_void_p(), ctypes.c_size_t(0)
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(ctypes.c_void_p(side.cuda_stream), 2) == 0
    forward.forward(x, out=out, stream=side)
    assert rt.cudaStreamEndCapture(ctypes.c_void_p(side.cuda_stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0 and rt.cudaGraphDestroy(graph) == 0
    return n.value


def test_fused_layer_boundary_in_front_of_a_row_of_several_units(monkeypatch):
    # the first row left to the SpMM spans several units (27 tuples): it is multiplied from its first unit on, and its
    # arrival counter is zero again for the products that follow
    import torch
    from accelgcn import synth, sharded, gcn
    dev = require_cuda()
    monkeypatch.setenv("AGCN_SPMM_PIECE", "0")
    light, heavy = 128 * 80, 3
    n = light + heavy
    rng = np.random.default_rng(3)
    deg = np.concatenate([np.full(light, 8), np.full(heavy, n)])
    ip = torch.from_numpy(np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)).to(dev)
    ix = torch.from_numpy(np.concatenate([rng.integers(0, n, light * 8), np.tile(np.arange(n), heavy)]).astype(np.int32)).to(dev)
    v = torch.from_numpy((rng.random(int(deg.sum())) / np.repeat(deg, deg)).astype(np.float32)).to(dev)
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    x = sh.to_block(synth.features(n, 128, 7, dev))
    w = [synth.glorot(128, 128, 7, k, dev) for k in (1, 2)]
    plain = gcn.GcnForward(sh, w)
    want = plain.forward(x).clone()
    monkeypatch.setenv("AGCN_GCN_FUSED", "1")
    fused = gcn.GcnForward(sh, w)
    scale = float(want.abs().max())
    assert _captured_nodes(fused, x) > _captured_nodes(plain, x)
    for _ in range(3):
        got = fused.forward(x, out=torch.full_like(x, float("nan")))
        assert float((got - want).abs().max()) <= 2e-3 * scale
        assert torch.equal(plain.forward(x, out=torch.full_like(x, float("nan"))), want)
    fused.status(); plain.status()
    fused.close(); plain.close(); sh.close()


def test_forward_with_fused_layer_boundary(monkeypatch):
    # AGCN_GCN_FUSED=1: the light rows of the block take the fused kernel between the layers, the others
    # SpMM + GEMM; the result must agree with the plain forward (same arithmetic, another summation order)
    import torch
    from accelgcn import synth, degree_sort, sharded, gcn
    dev = require_cuda()
    monkeypatch.setenv("AGCN_SPMM_PIECE", "0")             # plans whose tuples are cut do without the fused kernel
    g = synth.make_config(5, dev, 0.002)
    _, ip, ix, v = degree_sort.degree_sort_device(g.indptr, g.indices, g.vals)
    x = synth.features(g.n, 128, 1005, dev)
    w1, w2 = synth.glorot(128, 128, 1005, 8, dev), synth.glorot(128, 128, 1005, 9, dev)
    sh = sharded.ShardedSpmm(ip, ix, v, 0, 1)
    xb = sh.to_block(x)
    plain = gcn.GcnForward(sh, [w1, w2])
    want = plain.forward(xb).clone()
    torch.cuda.synchronize()
    plain.status()
    plain_nodes, plain_paired = _captured_nodes(plain, xb), plain.paired()
    plain.close()
    monkeypatch.setenv("AGCN_GCN_FUSED", "1")
    fused = gcn.GcnForward(sh, [w1, w2])
    got = fused.forward(xb)
    torch.cuda.synchronize()
    fused.status()
    assert plain_paired == (g.n >= 32_768) and not fused.paired()
    assert _captured_nodes(fused, xb) > plain_nodes        # the fused path is really taken at this size
    scale = float(want.abs().max())
    assert float((got - want).abs().max()) <= 2e-3 * scale
    fused.close(); sh.close()


def test_fused_layer_reports_a_column_out_of_range():
    import torch
    from accelgcn import gemm, synth, AccelGcnError
    dev = require_cuda()
    ip = torch.tensor([0, 2, 3], dtype=torch.int32, device=dev)
    ix = torch.tensor([1, 50, 7], dtype=torch.int32, device=dev)          # 50 is outside the 50 rows of Z1
    v = torch.ones(3, device=dev)
    z1 = synth.features(50, 128, 3, dev)
    w = torch.eye(128, device=dev)
    with pytest.raises(AccelGcnError, match="status 4"):
        gemm.gcn_fused_layer(ip, ix, v, z1, w, 2)
    ix[1] = 49
    got = gemm.gcn_fused_layer(ip, ix, v, z1, w, 2)                        # the device is fine: the next call succeeds
    want = torch.relu(torch.stack([z1[1] + z1[49], z1[7]]))
    assert torch.allclose(got, want, rtol=2e-3, atol=2e-3)
