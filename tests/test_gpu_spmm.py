"""SpMM parity on the GPU: the C ABI (through yitu_b200.ops / YiTu_GNN_kernel) against the CPU checker."""
import numpy as np
import pytest
import torch

from conftest import assert_close, random_csr

pytestmark = pytest.mark.gpu


def _dev(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    if dtype is not None:
        t = t.to(dtype)
    return t.cuda()


@pytest.mark.parametrize("D", [1, 3, 16, 20, 32, 48, 64, 100, 128, 200, 256, 512, 640])
@pytest.mark.parametrize("mode", ["none", "node", "edge"])
@pytest.mark.parametrize("kernel", ["auto", "rows", "stream"])
def test_spmm_modes_and_widths(oracle, monkeypatch, D, mode, kernel):
    from yitu_b200 import ops
    if kernel != "auto" and not 64 < D <= 256:
        pytest.skip("one kernel form for this width")
    monkeypatch.setenv("YITU_SPMM_STREAM", {"auto": "1", "rows": "0", "stream": "2"}[kernel])
    rng = np.random.default_rng(D * 7 + len(mode))
    n_rows, n_cols = 211, 173
    indptr, indices = random_csr(rng, n_rows, n_cols, density=0.05, hubs=3, hub_deg=150)
    x = rng.standard_normal((n_cols, D)).astype(np.float32)
    nd = rng.uniform(0.1, 1.0, n_rows).astype(np.float32)
    ns = rng.uniform(0.1, 1.0, n_cols).astype(np.float32)
    vals = rng.standard_normal(indices.shape[0]).astype(np.float32)
    rs = rng.uniform(0.5, 2.0, n_rows).astype(np.float32)
    kw_o = dict(wmode={"none": oracle.W_NONE, "node": oracle.W_NODE, "edge": oracle.W_EDGE}[mode])
    kw_g = dict(mode={"none": ops.W_NONE, "node": ops.W_NODE, "edge": ops.W_EDGE}[mode])
    if mode == "node":
        kw_o.update(norm_dst=nd, norm_src=ns)
        kw_g.update(norm_dst=_dev(nd), norm_src=_dev(ns))
    if mode == "edge":
        kw_o.update(values=vals)
        kw_g.update(edge_values=_dev(vals))
    ref = oracle.spmm(indptr, indices, x, row_scale=rs, alpha=0.5, **kw_o)
    for chunk in (0, 32, 512):  # no hub plan / every hub row split / default
        for ptr_dtype in (torch.int32, torch.int64):
            g = ops.PreparedGraph(_dev(indptr, ptr_dtype), _dev(indices), n_cols)
            got = ops.spmm(g, _dev(x), row_scale=_dev(rs), alpha=0.5, chunk_edges=chunk, **kw_g)
            assert_close(got.cpu().numpy(), ref, what="spmm D=%d %s chunk=%d" % (D, mode, chunk))


def test_spmm_accumulate_and_determinism(oracle):
    from yitu_b200 import ops
    rng = np.random.default_rng(5)
    indptr, indices = random_csr(rng, 300, 300, density=0.1, hubs=2, hub_deg=280)
    x = rng.standard_normal((300, 64)).astype(np.float32)
    base = rng.standard_normal((300, 64)).astype(np.float32)
    g = ops.PreparedGraph(_dev(indptr), _dev(indices), 300)
    out = _dev(base).clone()
    ops.spmm(g, _dev(x), out=out, accumulate=True, alpha=2.0, chunk_edges=64)
    ref = oracle.spmm(indptr, indices, x, alpha=2.0, out=base)
    assert_close(out.cpu().numpy(), ref, what="accumulate")
    a = ops.spmm(g, _dev(x), chunk_edges=64)
    b = ops.spmm(g, _dev(x), chunk_edges=64)
    assert torch.equal(a, b), "hub-split SpMM must be run-to-run identical (no float atomics)"


def test_empty_graph_and_empty_rows(oracle):
    from yitu_b200 import ops
    indptr = np.zeros(6, dtype=np.int32)
    indices = np.zeros(0, dtype=np.int32)
    g = ops.PreparedGraph(_dev(indptr), _dev(indices), 4)
    out = ops.spmm(g, torch.randn(4, 32, device="cuda"))
    assert out.shape == (5, 32) and float(out.abs().max()) == 0.0
    g0 = ops.PreparedGraph(_dev(np.zeros(1, dtype=np.int32)), _dev(indices), 4)
    assert ops.spmm(g0, torch.randn(4, 8, device="cuda")).shape == (0, 8)


def _csr_from_degrees(rng, degs, n_cols):
    rows = [np.sort(rng.choice(n_cols, size=int(k), replace=False)).astype(np.int32) for k in degs]
    indptr = np.zeros(len(degs) + 1, dtype=np.int64)
    indptr[1:] = np.cumsum([len(r) for r in rows])
    indices = np.concatenate(rows) if rows else np.zeros(0, dtype=np.int32)
    return indptr, indices.astype(np.int32)


STREAM_PATTERNS = {
    # runs of empty rows at the start, in the middle and at the end of 16-row batches
    "empty_runs": [0] * 5 + [3, 0, 0, 7, 1] + [0] * 20 + [40, 0, 33, 0, 0, 0] + [2] * 9 + [0] * 18,
    # rows that end exactly on 32-edge tile borders and on borders of the 4/8/16-edge gather groups
    "tile_borders": [32, 32, 64, 16, 16, 8, 8, 8, 8, 4, 4, 96, 1, 31, 33, 63, 65],
    # hub rows (above the 64-edge chunk limit used below) inside batches, adjacent to each other and at the ends
    "hubs_inside": [70, 3, 0, 200, 130, 5, 1] + [2] * 12 + [300] + [1] * 30 + [65, 64, 66],
    "single_row": [5],
    "only_empty": [0] * 37,
    "one_long_row_no_plan": [1000],
}


@pytest.mark.parametrize("pattern", sorted(STREAM_PATTERNS))
@pytest.mark.parametrize("D", [68, 96, 100, 128, 136, 256])
def test_stream_kernel_row_patterns(oracle, monkeypatch, pattern, D):
    """The edge-stream SpMM (warp = batch of consecutive rows walked as one edge stream) on row patterns that put
    every bookkeeping branch to work: empty rows anywhere in a batch, rows ending on tile / group borders, hub rows
    stepped over inside a batch, accumulate mode with and without an epilogue, every batch size and unroll."""
    from yitu_b200 import ops
    rng = np.random.default_rng(len(pattern) * 131 + D)
    n_cols = 1100
    degs = STREAM_PATTERNS[pattern]
    indptr, indices = _csr_from_degrees(rng, degs, n_cols)
    n_rows = len(degs)
    x = rng.standard_normal((n_cols, D)).astype(np.float32)
    vals = rng.standard_normal(indices.shape[0]).astype(np.float32)
    nd = rng.uniform(0.1, 1.0, n_rows).astype(np.float32)
    ns = rng.uniform(0.1, 1.0, n_cols).astype(np.float32)
    base = rng.standard_normal((n_rows, D)).astype(np.float32)
    bias = rng.standard_normal(D).astype(np.float32)
    chunk = 0 if pattern == "one_long_row_no_plan" else 64
    ref_edge = oracle.spmm(indptr, indices, x, wmode=oracle.W_EDGE, values=vals)
    ref_node = oracle.spmm(indptr, indices, x, wmode=oracle.W_NODE, norm_dst=nd, norm_src=ns)
    ref_acc = oracle.spmm(indptr, indices, x, alpha=0.5, out=base)
    ref_acc_epi = np.maximum(oracle.spmm(indptr, indices, x, out=base) + bias, 0)
    monkeypatch.setenv("YITU_SPMM_STREAM", "2")  # this kernel whatever the average row length
    for rows, eu in ((16, None), (8, None), (31, None), (16, 16 if D <= 128 else 8)):
        monkeypatch.setenv("YITU_SPMM_STREAM_ROWS", str(rows))
        if eu is None:
            monkeypatch.delenv("YITU_SPMM_STREAM_EU", raising=False)
        else:
            monkeypatch.setenv("YITU_SPMM_STREAM_EU", str(eu))
        for ptr_dtype in (torch.int32, torch.int64):
            g = ops.PreparedGraph(_dev(indptr, ptr_dtype), _dev(indices), n_cols)
            tag = "stream %s D=%d rows=%d eu=%s" % (pattern, D, rows, eu)
            got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
            assert_close(got.cpu().numpy(), ref_edge, what=tag + " edge")
            got = ops.spmm(g, _dev(x), mode=ops.W_NODE, norm_dst=_dev(nd), norm_src=_dev(ns), chunk_edges=chunk)
            assert_close(got.cpu().numpy(), ref_node, what=tag + " node")
            out = _dev(base).clone()
            ops.spmm(g, _dev(x), out=out, accumulate=True, alpha=0.5, chunk_edges=chunk)
            assert_close(out.cpu().numpy(), ref_acc, what=tag + " accumulate")
            out = _dev(base).clone()
            ops.spmm(g, _dev(x), out=out, accumulate=True, bias=_dev(bias), activation="relu", chunk_edges=chunk)
            assert_close(out.cpu().numpy(), ref_acc_epi, what=tag + " accumulate+epilogue")
    # the split form of huge power-law graphs (hub chunks on the group kernel, every other row on the edge-stream kernel, one
    # reduction) and, with 1, whatever the dispatch takes for so few rows
    monkeypatch.delenv("YITU_SPMM_STREAM_ROWS", raising=False)
    monkeypatch.delenv("YITU_SPMM_STREAM_EU", raising=False)
    for form in ("3", "1"):
        monkeypatch.setenv("YITU_SPMM_STREAM", form)
        tag = "%s %s D=%d" % ("split" if form == "3" else "default", pattern, D)
        g = ops.PreparedGraph(_dev(indptr, torch.int64), _dev(indices), n_cols)
        got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
        assert_close(got.cpu().numpy(), ref_edge, what=tag + " edge")
        got = ops.spmm(g, _dev(x), mode=ops.W_NODE, norm_dst=_dev(nd), norm_src=_dev(ns), chunk_edges=chunk)
        assert_close(got.cpu().numpy(), ref_node, what=tag + " node")
        out = _dev(base).clone()
        ops.spmm(g, _dev(x), out=out, accumulate=True, alpha=0.5, chunk_edges=chunk)
        assert_close(out.cpu().numpy(), ref_acc, what=tag + " accumulate")
        out = _dev(base).clone()
        ops.spmm(g, _dev(x), out=out, accumulate=True, bias=_dev(bias), activation="relu", chunk_edges=chunk)
        assert_close(out.cpu().numpy(), ref_acc_epi, what=tag + " accumulate+epilogue")
    # the group kernel on the same inputs gives the same sums up to the order of the additions
    monkeypatch.setenv("YITU_SPMM_STREAM", "0")
    g = ops.PreparedGraph(_dev(indptr, torch.int32), _dev(indices), n_cols)
    got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
    assert_close(got.cpu().numpy(), ref_edge, what="rows-kernel %s D=%d" % (pattern, D))


GROUP_WIDTHS = [1, 2, 4, 5, 8, 9, 12, 16, 17, 20, 24, 32, 33, 36, 40, 41, 48, 49, 60, 64, 65, 72, 97, 100, 120, 128, 129, 132, 136, 260, 264, 520]


@pytest.mark.parametrize("D", GROUP_WIDTHS)
@pytest.mark.parametrize("degrees", ["short", "mixed"])
def test_group_kernel_dispatch_edges(oracle, monkeypatch, D, degrees):
    """Every width class of the group kernel (two widths around each border; 256-, 128- and 32-bit loads), with rows that
    end inside, at and behind a tile of ids, hub rows cut into chunks, and strided and misaligned outputs of the C ABI."""
    import ctypes as C
    from yitu_b200 import ops
    from yitu_b200._lib import SpmmArgs, check, lib
    monkeypatch.setenv("YITU_SPMM_STREAM", "0")
    rng = np.random.default_rng(D * 3 + len(degrees))
    n_cols = 400
    degs = [0, 1, 2, 3, 4, 5, 7, 8, 9, 0, 6] * 3 if degrees == "short" else \
        [0, 1, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 0, 129, 300, 2, 0, 7]
    indptr, indices = _csr_from_degrees(rng, degs, n_cols)
    n_rows = len(degs)
    x = rng.standard_normal((n_cols, D)).astype(np.float32)
    vals = rng.standard_normal(indices.shape[0]).astype(np.float32)
    bias = rng.standard_normal(D).astype(np.float32)
    base = rng.standard_normal((n_rows, D)).astype(np.float32)
    ref = oracle.spmm(indptr, indices, x, wmode=oracle.W_EDGE, values=vals)
    ref_acc = np.maximum(oracle.spmm(indptr, indices, x, alpha=0.5, out=base) + bias, 0)
    g = ops.PreparedGraph(_dev(indptr, torch.int32), _dev(indices), n_cols)
    for chunk in (0, 64, ops.OWN_CHUNKS):
        got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
        assert_close(got.cpu().numpy(), ref, what="group %s D=%d chunk=%s" % (degrees, D, chunk))
        out = _dev(base).clone()
        ops.spmm(g, _dev(x), out=out, accumulate=True, alpha=0.5, bias=_dev(bias), activation="relu", chunk_edges=chunk)
        assert_close(out.cpu().numpy(), ref_acc, what="group %s D=%d chunk=%s accumulate" % (degrees, D, chunk))
    # rows that start 4 / 16 bytes behind a 32-byte boundary, and strides wider than the rows
    for shift, pad in ((1, 3), (4, 4), (0, 8)):
        xs = torch.zeros(n_cols, D + pad, device="cuda").view(-1)
        xs = torch.cat([xs, xs.new_zeros(8)])[shift:shift + n_cols * (D + pad)].view(n_cols, D + pad)
        xs[:, :D] = _dev(x)
        out = torch.full((n_rows, D + pad), 7.0, device="cuda")
        a = SpmmArgs()
        a.graph, a.n_heads, a.n_feats, a.weight_mode, a.alpha = g.csr, 1, D, ops.W_EDGE, 1.0
        v = _dev(vals)
        a.edge_values, a.x, a.x_stride = ops._ptr(v), C.c_void_p(xs.data_ptr()), D + pad
        a.out, a.out_stride = ops._ptr(out), D + pad
        check(lib().yitu_spmm_csr_f32(C.byref(a), ops._stream(xs.device)))
        assert_close(out[:, :D].cpu().numpy(), ref, what="group %s D=%d shift=%d pad=%d" % (degrees, D, shift, pad))
        assert bool((out[:, D:] == 7.0).all())


@pytest.mark.parametrize("D", [1, 4, 7, 8, 16, 20, 24, 32, 40, 41, 64, 100, 128, 200, 256, 260, 320])
def test_rows_are_summed_in_the_order_they_are_stored(D):
    """A row that is not cut into chunks is summed edge after edge, rows of 33..64 floats in whole 32-byte slices in four
    interleaved sums.  (A schedule cuts longer rows by the graph's size, and sums their chunks apart.)"""
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(D)
    degs = torch.tensor([0, 1, 2, 3, 5, 8, 13, 31, 32, 33, 47, 64], device="cuda")
    indptr = torch.zeros(degs.numel() + 1, dtype=torch.int32, device="cuda")
    indptr[1:] = degs.cumsum(0).to(torch.int32)
    n_cols = 300
    indices = torch.randint(0, n_cols, (int(degs.sum()),), device="cuda", generator=gen).to(torch.int32)
    x = torch.randn(n_cols, D, device="cuda", generator=gen)
    g = ops.PreparedGraph(indptr, indices, n_cols)
    out = ops.spmm(g, x)
    four = 32 < D <= 64 and D % 8 == 0
    for r, deg in enumerate(degs.tolist()):
        rows = x[indices[int(indptr[r]):int(indptr[r]) + deg].long()]
        parts = []
        for s in range(4 if four else 1):
            a = torch.zeros(D, device="cuda")
            for row in rows[s::4 if four else 1]:
                a = a + row
            parts.append(a)
        ref = (parts[0] + parts[1]) + (parts[2] + parts[3]) if four else parts[0]
        assert torch.equal(out[r], ref), "D=%d, row of %d edges" % (D, deg)


def test_infinite_features_stay_infinite():
    """Lanes behind a row's last edge gather nothing, so an infinite feature sums to infinity and not to NaN."""
    from yitu_b200 import ops
    x = torch.randn(8, 64, device="cuda")
    x[3] = float("inf")
    g = ops.PreparedGraph(torch.tensor([0, 3, 4], dtype=torch.int32, device="cuda"),
                          torch.tensor([3, 1, 2, 5], dtype=torch.int32, device="cuda"), 8)
    out = ops.spmm(g, x)
    assert bool(torch.isinf(out[0]).all()) and torch.equal(out[1], x[5])


def test_kernel_module_matches_oracle_on_gcn_graph(oracle):
    """2-layer GCN forward of the small benchmark configuration, plus the other YiTu_GNN_kernel entry points."""
    from yitu_b200 import YiTu_GNN_kernel as K, graphs
    n = 16384
    indptr, indices, norm = graphs.gcn_small()
    x = graphs.randn_features(0, n, 128)
    w1 = graphs.glorot_uniform(11, 128, 64)
    w2 = graphs.glorot_uniform(12, 64, 16)
    ip, ix, nm = indptr.cuda(), indices.cuda(), norm.cuda()
    pp, p2n = K.build_part(32, indptr)
    pp, p2n = pp.int().cuda(), p2n.int().cuda()
    args = (ip, ix, nm, pp, p2n, 32, 32, 2)
    h1 = K.forward(x.cuda(), w1.cuda(), *args)[0]
    out = K.forward(torch.relu(h1), w2.cuda(), *args)[0]
    r1 = oracle.gcn_forward(x.numpy(), w1.numpy(), indptr.numpy(), indices.numpy(), norm.numpy())
    r2 = oracle.gcn_forward(np.maximum(r1, 0), w2.numpy(), indptr.numpy(), indices.numpy(), norm.numpy())
    assert_close(h1.cpu().numpy(), r1, what="gcn layer 1")
    assert_close(out.cpu().numpy(), r2, rtol=2e-5, what="gcn layer 2")

    # backward: true transpose by default; the reference's forward-CSR variant behind the flag
    d_out = graphs.randn_features(3, n, 64)
    d_in, d_w = K.backward(d_out.cuda(), x.cuda(), w1.cuda(), *args)
    rd_in, rd_w = oracle.gcn_backward(d_out.numpy(), x.numpy(), w1.numpy(), indptr.numpy(), indices.numpy(),
                                      norm.numpy(), transpose=True)
    assert_close(d_in.cpu().numpy(), rd_in, rtol=2e-5, what="gcn d_input")
    assert_close(d_w.cpu().numpy(), rd_w, rtol=2e-5, what="gcn d_weight")
    K.BACKWARD_USES_FORWARD_CSR = True
    try:
        d_in2, _ = K.backward(d_out.cuda(), x.cuda(), w1.cuda(), *args)
    finally:
        K.BACKWARD_USES_FORWARD_CSR = False
    rd_in2, _ = oracle.gcn_backward(d_out.numpy(), x.numpy(), w1.numpy(), indptr.numpy(), indices.numpy(),
                                    norm.numpy(), transpose=False)
    assert_close(d_in2.cpu().numpy(), rd_in2, rtol=2e-5, what="gcn d_input (forward CSR)")

    # SAG and GIN
    xs = x[:, :64].contiguous()
    sag = K.SAG(xs.cuda(), *args)
    assert_close(sag.cpu().numpy(), oracle.spmm(indptr.numpy(), indices.numpy(), xs.numpy()), what="SAG")
    wg = graphs.glorot_uniform(13, 64, 32)
    gargs = (ip, ix, 0.5, pp, p2n, 32, 32, 2)
    o_gin, agg = K.forward_gin(xs.cuda(), wg.cuda(), *gargs)
    r_gin, r_agg = oracle.gin_forward(xs.numpy(), wg.numpy(), indptr.numpy(), indices.numpy(), 0.5)
    assert_close(agg.cpu().numpy(), r_agg, what="gin agg")
    assert_close(o_gin.cpu().numpy(), r_gin, rtol=2e-5, what="gin out")
    dg = graphs.randn_features(4, n, 32)
    di, dw = K.backward_gin(dg.cuda(), agg, wg.cuda(), *gargs)
    rdi, rdw = oracle.gin_backward(dg.numpy(), r_agg, wg.numpy(), indptr.numpy(), indices.numpy(), 0.5)
    assert_close(di.cpu().numpy(), rdi, rtol=2e-5, what="gin d_input")
    assert_close(dw.cpu().numpy(), rdw, rtol=2e-5, what="gin d_weight")


def test_input_contract():
    from yitu_b200 import YiTu_GNN_kernel as K
    x = torch.randn(4, 8)
    ip = torch.tensor([0, 1, 2, 3, 4], dtype=torch.int32).cuda()
    ix = torch.tensor([0, 1, 2, 3], dtype=torch.int32).cuda()
    d = torch.ones(4).cuda()
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        K.SAG(x, ip, ix, d, ip, ix, 32, 32, 2)
    with pytest.raises(RuntimeError, match="contiguous"):
        K.SAG(torch.randn(8, 4).cuda().t(), ip, ix, d, ip, ix, 32, 32, 2)


def test_graph_tables_bit_exact(oracle):
    from yitu_b200 import ops
    rng = np.random.default_rng(17)
    indptr, indices = random_csr(rng, 1500, 900, density=0.03, hubs=4, hub_deg=700)
    for ptr_dtype in (torch.int32, torch.int64):
        g = ops.PreparedGraph(_dev(indptr, ptr_dtype), _dev(indices), 900)
        t_ip, t_rows, t_perm = g.transpose()
        r_ip, r_rows, r_perm = oracle.csr_transpose(indptr, indices, 900)
        assert np.array_equal(t_ip.cpu().numpy().astype(np.int64), r_ip)
        assert np.array_equal(t_rows.cpu().numpy(), r_rows)
        assert np.array_equal(t_perm.cpu().numpy(), r_perm)
        for parts in (1, 2, 3, 8):
            b = ops.partition_rows(g, parts).cpu().numpy()
            assert np.array_equal(b, oracle.partition_rows(indptr, parts))
        plan = g.plan(64)
        deg = np.diff(indptr)
        exp_rows, exp_begin = [], []
        for r in np.nonzero(deg > 64)[0]:
            for j in range((deg[r] + 63) // 64):
                exp_rows.append(r)
                exp_begin.append(indptr[r] + 64 * j)
        assert plan[0].n_chunks == len(exp_rows)
        assert np.array_equal(plan[1].cpu().numpy(), np.asarray(exp_rows, dtype=np.int32))
        assert np.array_equal(plan[2].cpu().numpy(), np.asarray(exp_begin, dtype=np.int64))


def test_full_size_properties():
    """Benchmark-size graph (2^21 nodes, 2^26 sampled edges, 256 features): properties that need no CPU pass.
    unweighted A*1 = in-degree; linearity in x; hub-split and unsplit schedules agree."""
    from yitu_b200 import graphs, ops
    n = 1 << 21
    indptr, indices, values = graphs.spmm_rmat(device="cuda", n=n, e=1 << 26)
    g = ops.PreparedGraph(indptr, indices, n)
    deg = (indptr[1:] - indptr[:-1]).float()
    ones = torch.ones(n, 4, device="cuda")
    out = ops.spmm(g, ones)
    assert torch.equal(out[:, 0], deg), "A*1 must equal the in-degree exactly (integers < 2^24)"
    x1 = graphs.randn_features(1, n, 256, device="cuda")
    y1 = ops.spmm(g, x1, mode=ops.W_EDGE, edge_values=values)
    y1b = ops.spmm(g, x1, mode=ops.W_EDGE, edge_values=values, chunk_edges=0)
    scale = float(y1.abs().max())
    assert float((y1 - y1b).abs().max()) <= 2e-5 * scale
    y2 = ops.spmm(g, x1 * 2.0, mode=ops.W_EDGE, edge_values=values)
    assert torch.equal(y2, y1 * 2.0), "scaling x by 2 is exact in binary floating point"
    # transposed product: <A x, y> == <x, A^T y> within reduction tolerance (float64 dots)
    gt = g.t_prepared()
    t_perm = g.transpose()[2]
    yv = graphs.randn_features(2, n, 256, device="cuda")
    aty = ops.spmm(gt, yv, mode=ops.W_EDGE, edge_values=values, edge_perm=t_perm)
    lhs = float((y1.double() * yv.double()).sum())
    rhs = float((x1.double() * aty.double()).sum())
    assert abs(lhs - rhs) <= 1e-5 * max(abs(lhs), abs(rhs), 1.0) + 1e-2


def _rows_truth_f64(indptr, indices, values, x, rows):
    """float64 aggregation of a few destination rows, straight from the definition."""
    out = []
    for r in rows.tolist():
        b, e = int(indptr[r]), int(indptr[r + 1])
        cols = indices[b:e].long()
        w = values[b:e].double() if values is not None else torch.ones(e - b, dtype=torch.float64, device=x.device)
        out.append((w[:, None] * x[cols].double()).sum(0))
    return torch.stack(out)


def test_full_size_sampled_rows_against_float64():
    """Benchmark-size SpMM (2^21 nodes, 63.5 M edges, 256 features): 300 sampled destination rows, among them the
    longest hub rows, forward and transposed, against float64 sums at the 1e-5 bar."""
    from yitu_b200 import graphs, ops
    n = 1 << 21
    indptr, indices, values = graphs.spmm_rmat(device="cuda", n=n, e=1 << 26)
    g = ops.PreparedGraph(indptr, indices, n)
    x = graphs.randn_features(1, n, 256, device="cuda")
    y = ops.spmm(g, x, mode=ops.W_EDGE, edge_values=values)
    deg = indptr[1:] - indptr[:-1]
    gen = torch.Generator(device="cpu").manual_seed(0)
    rows = torch.cat([torch.topk(deg, 20).indices.cpu(), torch.randint(0, n, (280,), generator=gen)])
    truth = _rows_truth_f64(indptr, indices, values, x, rows)
    scale = float(truth.abs().max())
    err = (y[rows.cuda()].double() - truth).abs()
    assert float((err - 1e-5 * (truth.abs() + scale)).max()) <= 0, "forward rows off by %g" % float(err.max())
    # transposed product over the CSC built on the device
    gt = g.t_prepared()
    t_indptr, t_rows, t_perm = g.transpose()
    yt = ops.spmm(gt, x, mode=ops.W_EDGE, edge_values=values, edge_perm=t_perm)
    out_deg = t_indptr[1:] - t_indptr[:-1]
    cols = torch.cat([torch.topk(out_deg, 20).indices.cpu(), torch.randint(0, n, (280,), generator=gen)])
    truth_t = _rows_truth_f64(t_indptr, t_rows, values[t_perm.long()], x, cols)
    scale_t = float(truth_t.abs().max())
    err_t = (yt[cols.cuda()].double() - truth_t).abs()
    assert float((err_t - 1e-5 * (truth_t.abs() + scale_t)).max()) <= 0, "transposed rows off by %g" % float(err_t.max())


def test_partitioned_config_on_one_gpu_sampled_rows_against_float64():
    """The 8-GPU configuration's graph on one GPU: R-MAT 2^24 nodes, 2^29 sampled edges, int64 row pointers,
    weights 1/in-degree, 128 features (2^31 feature elements: element offsets use all 32 bits).  Sampled destination
    rows in float64 - the longest rows, rows whose sources lie at the very end of the feature matrix, and random
    ones - plus the exact identities A*1 = in-degree and (A/deg)*1 = 1."""
    from yitu_b200 import graphs, ops
    n, d = 1 << 24, 128
    indptr, indices, values = graphs.spmm_partitioned(device="cuda", n=n, e=1 << 29)
    assert indptr.dtype == torch.int64
    g = ops.PreparedGraph(indptr, indices, n)
    deg = indptr[1:] - indptr[:-1]
    ones = torch.ones(n, 4, device="cuda")
    assert torch.equal(ops.spmm(g, ones)[:, 0], deg.float()), "A*1 must equal the in-degree exactly"
    del ones
    x = graphs.randn_features(1, n, d, device="cuda")
    y = ops.spmm(g, x, mode=ops.W_EDGE, edge_values=values)
    gen = torch.Generator(device="cpu").manual_seed(0)
    # destination rows of the edges whose source id is largest (the last rows of x, offsets just below 2^31)
    far = torch.topk(indices.long(), 64).indices
    far_rows = (torch.searchsorted(indptr, far, right=True) - 1).cpu()
    assert int(indices.max()) * d + d > (1 << 30), "the sample must reach the upper half of the offset range"
    rows = torch.cat([torch.topk(deg, 16).indices.cpu(), far_rows, torch.randint(0, n, (240,), generator=gen)]).unique()
    truth = _rows_truth_f64(indptr, indices, values, x, rows)
    scale = float(truth.abs().max())
    err = (y[rows.cuda()].double() - truth).abs()
    assert float((err - 1e-5 * (truth.abs() + scale)).max()) <= 0, "rows off by %g" % float(err.max())
    from conftest import record_error
    big = truth.abs() >= 0.01 * scale
    record_error("partitioned-config-1gpu", float(err.max()) / scale, float((err[big] / truth.abs()[big]).max()))


def test_no_chunks_means_no_schedule():
    """chunk_edges 0 and None: rows are not split and no schedule is built, so a first call may be captured in a CUDA graph."""
    from yitu_b200 import ops
    n, deg = 50, 700
    indptr = torch.arange(0, (n + 1) * deg, deg, dtype=torch.int32, device="cuda")
    indices = torch.randint(0, n, (n * deg,), device="cuda").to(torch.int32)
    x, q, k = torch.randn(n, 2, 8, device="cuda"), torch.randn(n, 2, device="cuda"), torch.randn(n, 2, device="cuda")
    attn = torch.rand(n * deg, 2, device="cuda")
    grad = torch.randn(n, 2, 8, device="cuda")

    def calls(g, chunk):
        gat = ops.gat_fwd(g, q, k, x, chunk_edges=chunk)
        ops.gat_bwd(g, q, k, x, *gat, grad, chunk_edges=chunk)
        ops.edge_dot(g, grad, x, chunk_edges=chunk)
        ops.spmm_bwd(g, attn, x, grad, chunk_edges=chunk)
        ops.edge_softmax_bwd(g, q[None], k, ops.edge_softmax_fwd(g, q[None], k, chunk_edges=chunk), attn, chunk_edges=chunk)
        return ops.spmm(g, x, chunk_edges=chunk)

    want = calls(ops.PreparedGraph(indptr, indices, n), 0)
    for chunk in (0, None):
        g = ops.PreparedGraph(indptr, indices, n)
        g.t_prepared()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = calls(g, chunk)
        assert not g._plans and not g.t_prepared()._plans
        graph.replay()
        assert torch.equal(out, want)


@pytest.mark.parametrize("D", [1, 8, 24, 41, 64, 100, 128, 200, 256, 264])
def test_node_weights_do_not_depend_on_the_graph_around_a_row(monkeypatch, D):
    """norm_dst[r] * sum of norm_src[c] x[c] is rounded the same way in every graph and kernel, and the group kernel leaves a row
    without edges at 0 even where its factor is infinite (1 / sqrt(0))."""
    from yitu_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(D)
    degs = torch.tensor([3, 0, 30, 7, 0, 60], device="cuda")
    n_cols = 200
    indices = torch.randint(0, n_cols, (int(degs.sum()),), device="cuda", generator=gen).to(torch.int32)
    x, ns = torch.randn(n_cols, D, device="cuda", generator=gen), torch.rand(n_cols, device="cuda", generator=gen)
    nd = torch.rand(degs.numel(), device="cuda", generator=gen)
    results = []
    for stream in ("0", "1", "2"):
        monkeypatch.setenv("YITU_SPMM_STREAM", stream)
        for pad in (0, 600):  # empty rows behind: the average row of the graph is short or long
            indptr = torch.zeros(degs.numel() + pad + 1, dtype=torch.int32, device="cuda")
            indptr[1:] = torch.cat([degs, degs.new_zeros(pad)]).cumsum(0).to(torch.int32)
            g = ops.PreparedGraph(indptr, indices, n_cols)
            norm = torch.cat([nd, nd.new_ones(pad)])
            norm[indptr[1:] == indptr[:-1]] = float("inf") if stream == "0" else 1.0
            results.append(ops.spmm(g, x, mode=ops.W_NODE, norm_dst=norm, norm_src=ns)[:degs.numel()])
            assert float(results[-1][degs == 0].abs().max()) == 0.0
    for r in results[1:]:
        assert torch.equal(r, results[0])


@pytest.mark.parametrize("D", [1, 4, 8, 12, 32, 41, 48, 64, 96, 128, 200, 256, 264])
def test_long_rows_in_pieces(oracle, monkeypatch, D):
    """Rows whose edges do not fit 32 bits are walked in pieces; here the pieces are 64 edges, so that rows end inside, at and
    behind a piece, next to rows of one piece and to chunks of a schedule."""
    from yitu_b200 import ops
    monkeypatch.setenv("YITU_SPMM_STREAM", "0")
    rng = np.random.default_rng(D)
    n_cols = 700
    indptr, indices = _csr_from_degrees(rng, [0, 1, 63, 64, 65, 128, 129, 3, 300, 500, 0, 640, 7], n_cols)
    x, vals = rng.standard_normal((n_cols, D)).astype(np.float32), rng.standard_normal(indices.shape[0]).astype(np.float32)
    g = ops.PreparedGraph(_dev(indptr, torch.int64), _dev(indices), n_cols)
    for chunk in (0, 256):
        whole = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
        monkeypatch.setenv("YITU_SPMM_PIECE", "64")
        got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
        monkeypatch.delenv("YITU_SPMM_PIECE")
        assert torch.equal(got, whole)
        assert_close(got.cpu().numpy(), oracle.spmm(indptr, indices, x, wmode=oracle.W_EDGE, values=vals), what="pieces D=%d" % D)


def test_plan_of_no_argument():
    """plan() is the schedule of chunks of 512 edges, and all that the operators need to be captured without a call before."""
    from yitu_b200 import ops
    n, deg = 300, 600
    indptr = torch.arange(0, (n + 1) * deg, deg, dtype=torch.int32, device="cuda")
    indices = torch.randint(0, n, (n * deg,), device="cuda").to(torch.int32)
    x = torch.randn(n, 32, device="cuda")
    want = ops.spmm(ops.PreparedGraph(indptr, indices, n), x)
    g = ops.PreparedGraph(indptr, indices, n)
    assert g.chunk_edges() < 512 and g.plan()[0].chunk_edges == 512 and g.plan()[0].n_chunks == 2 * n
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.spmm(g, x)
    graph.replay()
    assert torch.equal(out, want)


def test_an_explicit_chunk_length_builds_one_schedule():
    """Only plan() builds the operators' own schedule along; a call that names its chunk length builds that one."""
    from yitu_b200 import ops
    n, deg = 300, 600
    indptr = torch.arange(0, (n + 1) * deg, deg, dtype=torch.int32, device="cuda")
    indices = torch.randint(0, n, (n * deg,), device="cuda").to(torch.int32)
    x = torch.randn(n, 32, device="cuda")
    for chunk in (64, 512):
        g = ops.PreparedGraph(indptr, indices, n)
        ops.spmm(g, x, chunk_edges=chunk)
        assert list(g._plans) == [chunk]


@pytest.mark.parametrize("D", [1, 4, 8, 16, 20, 32, 41, 48, 50, 64, 72, 100, 101, 128, 200, 256])
def test_few_long_rows(oracle, D):
    """The deeper forms that graphs of few, evenly long rows take (64 edges per row on average), with and without chunks."""
    from yitu_b200 import ops
    rng = np.random.default_rng(D)
    n_cols = 300
    indptr, indices = _csr_from_degrees(rng, [64, 65, 95, 96, 97, 70, 0, 1, 128, 130, 200, 31, 33, 66], n_cols)
    assert indices.size >= 64 * (indptr.size - 1)
    x, vals = rng.standard_normal((n_cols, D)).astype(np.float32), rng.standard_normal(indices.shape[0]).astype(np.float32)
    bias, base = rng.standard_normal(D).astype(np.float32), rng.standard_normal((indptr.size - 1, D)).astype(np.float32)
    ref = oracle.spmm(indptr, indices, x, wmode=oracle.W_EDGE, values=vals)
    ref_acc = np.maximum(oracle.spmm(indptr, indices, x, alpha=0.5, out=base) + bias, 0)
    for dtype in (torch.int32, torch.int64):
        g = ops.PreparedGraph(_dev(indptr, dtype), _dev(indices), n_cols)
        for chunk in (0, 64, ops.OWN_CHUNKS):
            got = ops.spmm(g, _dev(x), mode=ops.W_EDGE, edge_values=_dev(vals), chunk_edges=chunk)
            assert_close(got.cpu().numpy(), ref, what="few-long-rows D=%d chunk=%s" % (D, chunk))
            out = _dev(base).clone()
            ops.spmm(g, _dev(x), out=out, accumulate=True, alpha=0.5, bias=_dev(bias), activation="relu", chunk_edges=chunk)
            assert_close(out.cpu().numpy(), ref_acc, what="few-long-rows D=%d chunk=%s accumulate" % (D, chunk))
