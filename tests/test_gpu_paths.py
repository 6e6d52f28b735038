"""Branches of the host and kernel dispatch, each at the sizes where it can go wrong, against the other entry points or
the oracle."""
import ctypes
import re
import weakref

import numpy as np
import pytest
import torch

from conftest import graph_nodes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg(lib_built):
    assert torch.cuda.is_available()
    import llama_cl_b200

    return llama_cl_b200


@pytest.mark.parametrize("rows", [1, 8, 9])
def test_host_fc_in_place_and_copied(pkg, rows):
    """Up to 8 rows the kernels work on the pinned buffers themselves, beyond that on copies: the same FC either way."""
    g = torch.Generator().manual_seed(rows)
    W = (torch.randn(1003, 640, generator=g) * 0.02).cuda()
    wq = pkg.llmops.offline_FC_quant_Q4A(W, qtype="q4_1", group_k=128)
    fc = pkg.host.HostFC(wq, 1003, max_rows=16)
    for _ in range(3):  # captured on the first call, replayed with new inputs afterwards
        x = torch.randn(1, rows, 640, generator=g)
        want = pkg.llmops.fc_Q4A(x.cuda(), wq, 1003).cpu()
        assert torch.equal(fc(x), want)


@pytest.mark.parametrize("rows", [1, 9])
def test_host_fc_refuses_unfit_weights(pkg, rows):
    """A slice of a packed tensor has the pitch of the whole; unsigned bytes are no packed tensor: both are refused."""
    full = torch.zeros(8, 16, 640, dtype=torch.int8, device="cuda")
    for wq, text in ((full[:, 4:12], "dense row-major"), (full.view(torch.uint8), r"is<int8>\(3\)")):
        for graph in (True, False):
            with pytest.raises(RuntimeError, match=text):
                fc = pkg.host.HostFC(wq, 256, max_rows=16, graph=graph)
                fc(torch.zeros(1, rows, fc.K))


def test_host_fc_in_place_forms(pkg):
    """The in-place path without a graph, without waiting, on given streams, two at once and as a group."""
    ops, HostFC = pkg.llmops, pkg.host.HostFC
    g = torch.Generator().manual_seed(6)
    shapes = [(300, 1024), (1003, 640)]
    ws = [ops.offline_FC_quant_Q4A((torch.randn(*s, generator=g) * 0.02).cuda(), qtype="q4_0") for s in shapes]
    xs = [[torch.randn(1, rows, K, generator=g) for _, K in shapes] for rows in (1, 8, 3, 1)]
    want = [[ops.fc_Q4A(x.cuda(), w, n).cpu() for x, w, (n, _) in zip(row, ws, shapes)] for row in xs]
    for graph in (True, False):
        fcs = [HostFC(w, n, graph=graph, stream=torch.cuda.Stream()) for w, (n, _) in zip(ws, shapes)]
        for row, ys in zip(xs, want):
            got = [f(x, sync=False) for f, x in zip(fcs, row)]
            for f in fcs:
                f.stream.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, ys))
            assert all(torch.equal(f(x), y) for f, x, y in zip(fcs, row, ys))
    group = pkg.host.HostFCGroup([HostFC(w, n) for w, (n, _) in zip(ws, shapes)])
    for row, ys in zip(xs, want):
        assert all(torch.equal(a, b) for a, b in zip(group(row), ys))


def test_host_fc_with_a_small_workspace_copies(pkg):
    """A workspace without room for the quantizer's codes: the kernel would read the host buffer once per cluster, so the
    activations are copied."""
    g = torch.Generator().manual_seed(5)
    wq = pkg.llmops.offline_FC_quant_Q4A((torch.randn(300, 1024, generator=g) * 0.02).cuda())
    x = torch.randn(1, 4, 1024, generator=g)
    size = pkg._cabi.lib().q4fc_fc_workspace_bytes(4, 1024, 300, 1, 32)
    for nbytes in (size - 256, size):
        fc = pkg.host.HostFC(wq, 300, workspace=pkg.llmops.Workspace(nbytes, wq.device))
        assert fc._reads_host(4) == (nbytes == size)
        assert torch.equal(fc(x), pkg.llmops.fc_Q4A(x.cuda(), wq, 300).cpu())


def test_host_fc_results_are_views_of_their_own(pkg):
    """What a caller does to the tensor that a call returned changes no later call's."""
    wq = pkg.llmops.offline_FC_quant_Q4A(torch.randn(96, 512).cuda())
    for graph in (True, False):
        fc = pkg.host.HostFC(wq, 96, graph=graph)
        x = torch.randn(1, 4, 512)
        y = fc(x)
        y.squeeze_(0).requires_grad_()
        z = fc(x)
        assert z is not y and z.shape == (1, 4, 96) and not z.requires_grad and z.data_ptr() == y.data_ptr()


def test_host_fc_refuses_overlapping_input(pkg):
    """Rows 1..4 of the staging buffer cannot be copied onto rows 0..3; rows 4..7 can, rows 0..3 need no copy."""
    g = torch.Generator().manual_seed(3)
    wq = pkg.llmops.offline_FC_quant_Q4A((torch.randn(96, 512, generator=g) * 0.02).cuda())
    fc = pkg.host.HostFC(wq, 96)
    x = torch.randn(1, 8, 512, generator=g)
    fc(x[:, :4])  # captured
    for lo in (0, 4):
        fc.x_staging(8).copy_(x)
        assert torch.equal(fc(fc.x_staging(8)[:, lo: lo + 4]), pkg.llmops.fc_Q4A(x[:, lo: lo + 4].cuda(), wq, 96).cpu())
    with pytest.raises(RuntimeError, match="single memory location"):
        fc(fc.x_staging(8)[:, 1:5])


def test_q8c_graph_outlives_a_larger_call(pkg):
    """A captured call keeps its scratch when a larger call on the stream needs another: the scratch is not handed out
    again, and the replay gives the captured call's result."""
    ops = pkg.llmops
    g = torch.Generator().manual_seed(0)
    w, s = pkg.c_ext.FC_quant_Q8C((torch.randn(200, 1024, generator=g) * 0.02).cuda())
    small, large = (torch.randn(1, rows, 1024, generator=g).cuda() for rows in (8, 2000))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        want = ops.FC_evaluate_Q8C(small, w, s, 200)
        key = (torch.cuda.current_device(), stream.cuda_stream)
        scratch = weakref.ref(ops._q8c_scratch[key])
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = ops.FC_evaluate_Q8C(small, w, s, 200)
        for rows in (9, 700, 2000):
            ops.FC_evaluate_Q8C(large[:, :rows].contiguous(), w, s, 200)
        assert scratch() is not None and ops._q8c_scratch[key] is not scratch()
        kept = sum(t.numel() for t in ops._retired if isinstance(t, torch.Tensor))
        assert kept < sum(t.numel() for t in ops._q8c_scratch.values())
        graph.replay()
    stream.synchronize()
    assert torch.equal(got, want)


def test_argument_forms(pkg):
    """Sizes are integers (fc_Q4A alone takes what int() takes); an unknown path is a KeyError unless an addend, which has
    one path, makes it meaningless."""
    ops = pkg.llmops
    W, x = torch.randn(64, 512).cuda(), torch.randn(1, 1, 512).cuda()
    wq, (w8, s8) = ops.offline_FC_quant_Q4A(W), pkg.c_ext.FC_quant_Q8C(W)
    for bad in (63.5, 64.0, "64", None):
        with pytest.raises(TypeError):
            ops.FC_evaluate_Q8C(x, w8, s8, bad)
    for bad in (32.0, "32", None):
        with pytest.raises(TypeError):
            ops.offline_FC_quant_Q4A(W, group_k=bad)
    for bad in (33, (1 << 32) + 32):
        with pytest.raises(RuntimeError):
            ops.offline_FC_quant_Q4A(W, group_k=bad)
    assert torch.equal(ops.FC_evaluate_Q8C(x, w8, s8, np.int64(60)), ops.FC_evaluate_Q8C(x, w8, s8, 60))
    assert torch.equal(ops.offline_FC_quant_Q4A(W, group_k=np.int64(32)), wq)
    want = ops.fc_Q4A(x, wq, 60)
    for n in (60.5, "60", np.int64(60)):
        assert torch.equal(ops.fc_Q4A(x, wq, n), want)
    bias = torch.zeros(60, device="cuda")
    for path in ("fast", None):
        with pytest.raises(KeyError):
            ops.fc_Q4A(x, wq, 60, path=path)
        assert torch.equal(ops.fc_Q4A(x, wq, 60, path=path, addend=bias), want)


def test_out_of_memory_is_torchs_own_error(pkg):
    """A result that no card holds (549 GB): torch.OutOfMemoryError, as torch.empty raises it, without a C++ trace."""
    op = pkg.ops.llmop_embedding_q8c(torch.randn(4, 4096, device="cuda"))
    with pytest.raises(torch.OutOfMemoryError) as e:
        op(torch.zeros(1 << 25, dtype=torch.int32, device="cuda"))
    assert "Exception raised from" not in str(e.value)


def test_stack_switches_its_graph_off(pkg):
    """use_graph = False after a captured token: the steps are enqueued one by one, as without a graph from the start."""
    H, I, V = 128, 256, 96
    g = torch.Generator().manual_seed(8)
    pack = lambda N, K: pkg.llmops.offline_FC_quant_Q4A((torch.randn(N, K, generator=g) * 0.02).cuda())
    layer = {k: pack(*s) for k, s in dict(q=(H, H), k=(H, H), v=(H, H), o=(H, H), gate=(I, H), up=(I, H), down=(H, I)).items()}
    st = pkg.stack.DecodeFCStack([layer], pack(V, H), hidden=H, intermediate=I, vocab=V)
    x = torch.randn(1, 1, H, generator=g).cuda()
    torch.cuda.synchronize()
    want = st.forward(x, sync=True).clone()
    assert torch.equal(st.forward(x, sync=True), want)
    calls, enqueue = [], st.enqueue
    st.enqueue = lambda: (calls.append(1), enqueue())
    st.use_graph = False
    assert torch.equal(st.forward(x, sync=True), want) and calls == [1]
    st.use_graph = True
    assert torch.equal(st.forward(x, sync=True), want) and calls == [1]


@pytest.mark.parametrize("device", [None, 0, "cuda", "cuda:0", torch.device("cuda"), torch.device("cuda", 0)])
def test_device_forms(pkg, device):
    pkg.llmops.check_device_status(device)


def test_status_word_texts(pkg):
    """The code of a wait that ran out (here: written from the host) is no bad embedding id, whichever letters it has."""
    ws = pkg.llmops.Workspace(4096, torch.device("cuda"))
    word = ws.buf[:4].view(torch.int32)
    for code in (b"PREF", b"RFUL", b"REMP", b"TPWT", b"CFUL", b"RXBQ"):
        word.fill_(int.from_bytes(code, "big"))
        with pytest.raises(RuntimeError, match=r"\(a bounded wait ran out\)"):
            ws.check()
        word.fill_(int.from_bytes(code, "big") | 0x80)
        with pytest.raises(RuntimeError, match=r"\(an embedding id was out of range; a bounded wait ran out\)"):
            ws.check()
        ws.check()  # cleared
    op = pkg.ops.llmop_embedding_q8c(torch.randn(10, 64, device="cuda"))
    op(torch.tensor([3, 10, -1], device="cuda"))
    with pytest.raises(RuntimeError, match=r"\(an embedding id was out of range\)"):
        pkg.llmops.check_device_status()
    pkg.llmops.check_device_status()


@pytest.mark.parametrize("qtype,G", [(0, 32), (1, 128)])
@pytest.mark.parametrize("rows", [1, 5, 8])
def test_few_rows_on_the_prefill_path(pkg, rows, qtype, G):
    """A workspace of exactly the stated size serves the prefill path at any row count, here and through HostFC."""
    ops, N, K = pkg.llmops, 96, 4100
    g = torch.Generator().manual_seed(rows)
    wq = ops.offline_FC_quant_Q4A((torch.randn(N, K, generator=g) * 0.02).cuda(), qtype=qtype, group_k=G)
    x = torch.zeros(1, rows, -(-K // G) * G)
    x[:, :, :K] = torch.randn(1, rows, K, generator=g)
    size = pkg._cabi.lib().q4fc_fc_workspace_bytes(rows, x.shape[2], N, qtype, G)
    ws = ops.Workspace(size, torch.device("cuda"))
    assert ws.nbytes == size
    got = ops.fc_Q4A(x.cuda(), wq, N, path="prefill", workspace=ws).cpu()
    ws.check()
    # 2 x 264 roundings of 2^-24 at most, which add up like a random walk: 1.4e-6 of the sum; a factor of ten on top
    want = ops.fc_Q4A(x.cuda(), wq, N, path="decode").cpu()
    assert (got - want).abs().max() <= 1.4e-5 * want.abs().max()
    assert torch.equal(pkg.host.HostFC(wq, N, max_rows=rows, path="prefill")(x), got)


@pytest.mark.parametrize("rows,N,K", [(65, 96, 4100), (128, 4096, 2080), (300, 12800, 1000)])
@pytest.mark.parametrize("qtype,G", [(0, 32), (1, 32), (1, 128)])
def test_many_rows_with_a_workspace_for_byte_codes(pkg, rows, N, K, qtype, G):
    """Room for a byte per activation code is enough: with group 32 for 64-row tiles, else for what a full workspace gives.  Less
    is refused."""
    ops = pkg.llmops
    g = torch.Generator(device="cuda").manual_seed(rows)
    wq = ops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype=qtype, group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    codes = rows * -(-K // G) * G
    size = pkg._cabi.lib().q4fc_fc_workspace_bytes(rows, K, N, qtype, G)
    whole = lambda nbytes: -(-nbytes // 256) * 256
    small = size - whole(2 * codes) + whole(codes) if G == 32 else size
    want = ops.fc_Q4A(x, wq, N)
    ws = ops.Workspace(small, torch.device("cuda"))
    got = ops.fc_Q4A(x, wq, N, workspace=ws)
    ws.check()
    # 2 x 129 roundings of 2^-24 at most on either side, as a random walk: 1.4e-6 of the largest sum; a factor of ten on top
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()
    if G == 32:
        assert gemm_launches(lambda: ops.fc_Q4A(x, wq, N, workspace=ws))[0][0] == ROWS64
    with pytest.raises(RuntimeError, match="workspace"):
        ops.fc_Q4A(x, wq, N, workspace=ops.Workspace(small - 256, torch.device("cuda")))


@pytest.mark.parametrize("rows,N,K", [
    (9, 4096, 512),     # one 16-row chunk
    (16, 130, 4128),    # a last stage with one K group; K divided unevenly; stripes that fill no tile of four
    (17, 97, 2080),     # two chunks, the second one row
    (64, 1000, 1056), (65, 1000, 1056),       # one 64-row tile, one row more
    (128, 20000, 160), (129, 10000, 160),     # 128-row tiles on every SM, one row more
    (33, 40, 33),       # less than a stage
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "q8c"])
def test_many_rows_on_tile_edges(pkg, oracle, fmt, rows, N, K):
    """Both tile sizes of the tensor-core FC and K divided by 1, 2, 4 and 8, against the oracle (the other divisions and
    long K: below).  At most 2 Kg <= 264 fp32 roundings of 2^-24 on either side of a sum, which add up like a random walk:
    1.4e-6 of its largest value; 2e-5 is a factor of ten and more on top."""
    check_many_rows(pkg, oracle, fmt, rows, N, K)


@pytest.mark.parametrize("rows,N,K", [
    # 64-row tiles; 29 stages, the last one group (which divisions there are, and that calls take them: test_every_division_of_k)
    (20, 11000, 3600), (17, 7550, 3600), (17, 6270, 3600), (17, 5370, 3600),
    (129, 10000, 1184),  # 128-row tiles on every SM: ten stages go around every ring, the last one group
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "signed32", "signed128", "q8c"])
def test_many_rows_divisions_and_long_k(pkg, oracle, fmt, rows, N, K):
    """Divided K, and tiles whose shared-memory rings wrap, in every format, against the oracle."""
    check_many_rows(pkg, oracle, fmt, rows, N, K)


@pytest.mark.parametrize("rows,N,K", [
    (129, 9500, 2080),    # 150 tiles of 128 rows on 148 SMs: two left, K divided by four, the last stage one group
    (150, 11648, 2080),   # 182 tiles, 34 left: K divided by three
    (6500, 300, 2080),    # 153 tiles, five left over three column tiles: the launch's rows of tiles wrap, the last is not full
    (20, 37900, 2084),    # 297 tiles of 64 rows on 296 places: one left, columns and k beyond the weights
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "signed32", "signed128", "q8c"])
def test_many_rows_last_tiles_divided(pkg, oracle, fmt, rows, N, K):
    """Tiles left over after whole rounds go in a launch of their own with K divided (tolerance as above)."""
    check_many_rows(pkg, oracle, fmt, rows, N, K, launches=3)  # the quantizer, whole rounds, the remainder


class _KernelNode(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def kernels_of(run):
    """The kernels of a captured call: name, and blocks of a cluster."""
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run()  # the stream's workspace
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            run()
    cu, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t()
    g = ctypes.c_void_p(graph.raw_cuda_graph())
    assert cu.cuGraphGetNodes(g, None, ctypes.byref(n)) == 0
    nodes, seen = (ctypes.c_void_p * n.value)(), []
    assert cu.cuGraphGetNodes(g, nodes, ctypes.byref(n)) == 0
    for node in map(ctypes.c_void_p, nodes):
        kernel, value, name = _KernelNode(), (ctypes.c_uint * 16)(), ctypes.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(node, ctypes.byref(kernel)) == 0
        assert cu.cuGraphKernelNodeGetAttribute(node, 4, value) == 0  # the cluster's dimension
        assert cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(kernel.func)) == 0
        seen.append((name.value, value[0]))
    return seen


ROWS64, ROWS128 = 64, 128  # rows of a tile: fc_prefill_kernel's (of Q8C also 128), and fc_prefill_wide_kernel's


def gemm_launches(run, moves=False):
    """What a call of the many-row FC launches behind the quantizer: for each kernel the rows of a tile and the blocks of a cluster;
    `moves`: also whether running sums move (of 64-row tiles 1 with at most 48 rows, else 2)."""
    seen = []
    for name, cluster in kernels_of(run):
        if tile := re.search(rb"fc_prefill_kernelILi\dELi\d+ELi(\d+)ELi(\d+)E", name):
            seen.append((int(tile[1]), cluster, int(tile[2])))
        elif tile := re.search(rb"fc_prefill_wide_kernelILi\dELi\d+ELb([01])E", name):
            seen.append((ROWS128, cluster, int(tile[1])))
    return [launch if moves else launch[:2] for launch in sorted(seen, key=lambda launch: launch[1])]


@pytest.mark.parametrize("rows,N,K,launches", [
    # few tiles: K by one to eight, the last stage not full; 69 tiles, which run at once by four on every card
    *[(20 if c % 2 else 50, 300, 512 * c + 300, [(ROWS64, c)]) for c in range(1, 9)], (31, 8707, 6030, [(ROWS64, 4)]),
    # a few more than two on each of 148 SMs
    *[(40, (296 + left) * 128 - 59, K, [(ROWS64, 1), (ROWS64, c)])
      for left, K, c in [(100, 4096, 2), (80, 4096, 3), (65, 4096, 4), (47, 4096, 5), (44, 4096, 6), (30, 3564, 7), (30, 4076, 8)]],
    # 128-row tiles, whole calls (the second, fourth, sixth and eighth: rows that are not there, more of them columns)
    *[(rows, tiles * 128 - 20, K, [(ROWS128, c)]) for c, (rows, tiles, K) in enumerate([
        (256, 74, 2000), (200, 35, 3000), (128, 38, 6500), (113, 31, 4000), (128, 23, 8000), (113, 22, 6500), (128, 14, 3900),
        (113, 15, 8000)], 1)],
    # and a few more than one on each SM
    *[(65, (148 + left) * 128 - 59, K, [(ROWS128, 1), (ROWS128, c)])
      for left, K, c in [(50, 4096, 2), (40, 4096, 3), (30, 4096, 4), (23, 4096, 5), (20, 4096, 6), (10, 3564, 7), (10, 4076, 8)]],
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "signed32", "signed128", "q8c"])
def test_every_division_of_k(pkg, fmt, rows, N, K, launches):
    """Every way to divide K, in either tile and for the last of many tiles, and that it is the one a call takes; against calls of
    at most eight rows, which other kernels serve: the same exact integers, other products and sums (tolerance as above)."""
    ops = pkg.llmops
    g = torch.Generator(device="cuda").manual_seed(rows + N + K)
    W, x = torch.randn(N, K, generator=g, device="cuda") * 0.02, torch.randn(1, rows, K, generator=g, device="cuda")
    if fmt == "q8c":
        if launches[0][0] == ROWS128:
            pytest.skip("Q8C has 128-row tiles of its own")
        w8, s8 = pkg.c_ext.FC_quant_Q8C(W)
        run, few = (lambda x: pkg.c_ext.FC_evaluate_Q8C(x, w8, s8, N),) * 2
    else:
        signed = isinstance(fmt, str)
        qtype, G = (0, int(fmt[6:])) if signed else fmt
        wq = ops.offline_FC_quant_Q4A(W, qtype=f"q4_{qtype}", group_k=G)
        run = lambda x: ops.fc_Q4A(x, wq, N, nibble_signed=signed)
        few = lambda x: ops.fc_Q4A(x, wq, N, nibble_signed=signed, path="decode")
    del W
    got = run(x)
    assert torch.equal(got, run(x))  # fixed summation order
    want = torch.cat([few(part.contiguous()) for part in x.split(8, dim=1)], dim=1)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()
    if fmt != "q8c" or N > 1000:  # (which leaves small problems to its own kernel)
        assert gemm_launches(lambda: run(x)) == launches
    ops.check_device_status()


@pytest.mark.parametrize("rows,N,K,launch", [
    (20, 40 * 128 - 20, 7600, (ROWS64, 6, 1)), (48, 40 * 128 - 20, 7600, (ROWS64, 6, 1)),  # 40 tiles by six instead of by seven
    (49, 40 * 128 - 20, 7600, (ROWS64, 6, 2)), (64, 40 * 128 - 20, 7600, (ROWS64, 6, 2)),
    (128, 36 * 128 - 20, 6500, (ROWS128, 3, 1)), (100, 36 * 128 - 20, 6500, (ROWS128, 3, 1)),  # 72 of 64 rows by four
    (20, 97 * 128, 1500, None),  # group 128: undivided instead of by three, two moves
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "signed32", "signed128"])
def test_running_sums_that_move(pkg, fmt, rows, N, K, launch):
    """Where K is divided by less than fills the GPU, the running sums move in between: each place they move to (tolerance as
    above)."""
    ops, signed = pkg.llmops, isinstance(fmt, str)
    qtype, G = (0, int(fmt[6:])) if signed else fmt
    g = torch.Generator(device="cuda").manual_seed(rows + N + K)
    wq = ops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype=f"q4_{qtype}", group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    x[0, 3], x[0, 5, 7], x[0, 9, 1], x[0, 10, 2] = 0, 1e6, float("inf"), float("nan")
    run = lambda x, path=None: ops.fc_Q4A(x, wq, N, nibble_signed=signed, **({"path": path} if path else {}))
    got, want = run(x), torch.cat([run(part.contiguous(), "decode") for part in x.split(8, dim=1)], dim=1)
    assert torch.equal(got.view(torch.int32), run(x).view(torch.int32))
    assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(got.isnan(), want.isnan())
    got, want = got.nan_to_num(0, 0, 0), want.nan_to_num(0, 0, 0)
    assert ((got - want).abs() <= 2e-5 * want.abs().amax(-1, keepdim=True)).all()
    seen = gemm_launches(lambda: run(x), moves=True)
    assert seen == [launch or ((ROWS64, 1, 1) if G == 128 else (ROWS64, 2, 1))]
    ops.check_device_status()


@pytest.mark.parametrize("rows,N,K", [(113, 18944, 640), (128, 18924, 640), (97, 18944, 3000), (65535 * 64 + 1, 20, 33)])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128)])
def test_wide_tiles_with_few_stages(pkg, fmt, rows, N, K):
    """128-row tiles with the fewest K stages that go in them, and beyond the rows that a grid of 64-row tiles has, where even
    less than one stage does; against calls that go in 64-row tiles (tolerance as above)."""
    ops, (qtype, G) = pkg.llmops, fmt
    g = torch.Generator(device="cuda").manual_seed(K)
    wq = ops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype=f"q4_{qtype}", group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    run = lambda x: ops.fc_Q4A(x, wq, N)
    got = run(x)
    few = 60 if rows < 1000 else 1 << 21
    want = torch.cat([run(part.contiguous()) for part in x.split(few, dim=1)], dim=1)
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()
    assert gemm_launches(lambda: run(x)) == [(ROWS128, 1)]
    assert gemm_launches(lambda: run(x[:, :few].contiguous()))[0][0] == ROWS64
    ops.check_device_status()


@pytest.mark.parametrize("rows,K,stripes,qtype,G,sharers", [
    (1, 4096, 140, 1, 32, 2), (1, 4096, 131, 1, 32, 4), (4, 4000, 290, 0, 32, 2),  # a round saved, none, a round
    (5, 2560, 288, 1, 128, 4), (6, 2730, 271, 1, 128, 4), (7, 2340, 138, 0, 128, 4),  # a round, but a second pass of the quantizer
])
def test_sharers_of_the_quantizer(pkg, rows, K, stripes, qtype, G, sharers):
    """Two CTAs share the quantizer instead of four only where the SMs so reached are worth its longer share."""
    g = torch.Generator(device="cuda").manual_seed(stripes)
    wq = pkg.llmops.offline_FC_quant_Q4A(torch.randn(stripes * 32, K, generator=g, device="cuda") * 0.02, qtype=qtype, group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    assert kernels_of(lambda: pkg.llmops.fc_Q4A(x, wq, stripes * 32))[0][1] == sharers


def fc_in_64_bits(oracle, wq, x, N, G):
    """Q4_0, signed nibbles, on the oracle's activation codes and scales, summed in 64 bits."""
    Ng, Kg, rows = wq.shape[0], wq.shape[1], x.shape[1]
    blocks = wq.view(torch.uint8).view(Ng, Kg, -1)
    nibbles = blocks[:, :, :16 * G].reshape(Ng, Kg, G // 8, 32, 4)
    weights = (torch.cat([nibbles & 15, nibbles >> 4], dim=-1).permute(1, 2, 4, 0, 3).reshape(Kg * G, Ng * 32) ^ 8).double() - 8
    scales = blocks[:, :, 16 * G:].contiguous().view(torch.float16).permute(1, 0, 2).reshape(Kg, Ng * 32).double()
    codes, d, _ = (torch.from_numpy(a).cuda().double() for a in oracle.restated.quant_x(x[0].cpu().numpy(), G))
    return ((codes * d.repeat_interleave(G, 1)) @ (weights * scales.repeat_interleave(G, 0)))[:, :N]


@pytest.mark.parametrize("rows,N,K,G,chain", [
    (49, 9384, 10740, 32, 84), (36, 9384, 10740, 32, 84), (20, 11441, 1900, 128, 5),     # 64-row tiles where few divisions of K are
    (128, 6000, 3000, 32, 32), (77, 3619, 10624, 32, 68), (90, 3520, 10310, 128, 17),  # the fastest; 128-row tiles
])
def test_many_rows_sums_are_as_exact_as_with_every_place_taken(pkg, oracle, rows, N, K, G, chain):
    """No running fp32 sum has more terms than `chain`: K groups over the times that two places on each of 148 SMs hold the
    call's 64-row tiles.  An addition rounds off 2.53e-8 of its result in the root mean square (2^-24 at most, evenly, mantissas
    spread logarithmically), so a random walk of L terms 2.53e-8 sqrt(L / 2) of the sum; the products and adding the parts count
    as four steps more.  3 % on top (seen: 0.2 % at most)."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    wq = pkg.llmops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype="q4_0", group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    want = fc_in_64_bits(oracle, wq, x, N, G)
    error = (pkg.llmops.fc_Q4A(x, wq, N, nibble_signed=True)[0] - want).norm() / want.norm()
    assert error <= 1.03 * 2.53e-8 * (chain / 2 + 4) ** 0.5


@pytest.mark.parametrize("stripes", [75, 77, 131, 133, 148, 149, 266, 296, 297])
@pytest.mark.parametrize("rows,K,qtype,G", [(1, 1000, 1, 32), (3, 2080, 0, 128), (1, 9000, 1, 128), (2, 4096, 0, 32)])
def test_decode_ctas_that_share_the_quantizer(pkg, stripes, rows, K, qtype, G):
    """Four or two CTAs to a share, CTAs without a stripe, one to three rounds of stripes: bit-equal to quantizing in front."""
    g = torch.Generator(device="cuda").manual_seed(stripes + K)
    N = stripes * 32 - 5
    wq = pkg.llmops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype=f"q4_{qtype}", group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    want = pkg.llmops.fc_Q4A_q8(pkg.llmops.quantize_activations(x, G), wq, N)
    assert torch.equal(pkg.llmops.fc_Q4A(x, wq, N, path="decode"), want)


@pytest.mark.parametrize("rows,N,K", [
    # 148 column tiles and more: whole tiles, the last columns and K groups not full, few K stages and more than the rings hold, rows
    # that end in each of a warp's four chunks (which calls go in 128-row tiles: test_every_division_of_k and the one behind it)
    (65, 18901, 33), (81, 18901, 96), (112, 18920, 224), (128, 18944, 1312), (129, 9473, 640), (185, 9473, 160),
    (128, 1024, 4096), (192, 1000, 4096), (129, 4096, 2080), (300, 1500, 4096), (128, 6000, 3000),  # K divided
])
@pytest.mark.parametrize("fmt", [(0, 32), (0, 128), (1, 32), (1, 128), "signed32", "signed128"])
def test_wide_tiles_against_64_row_tiles(pkg, fmt, rows, N, K):
    """More than 64 rows, in either tile, against calls of at most 64 rows, which go in 64-row tiles: the same codes and exact
    integers, products and sums in another order (tolerance as in test_many_rows_on_tile_edges, row by row).  Among the rows the ends of the range."""
    signed = isinstance(fmt, str)
    qtype, G = (0, int(fmt[6:])) if signed else fmt
    g = torch.Generator(device="cuda").manual_seed(rows + N + K)
    wq = pkg.llmops.offline_FC_quant_Q4A(torch.randn(N, K, generator=g, device="cuda") * 0.02, qtype=f"q4_{qtype}", group_k=G)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    x[0, 3], x[0, 5:8] = 0, x[0, 5:8] * torch.tensor([[1e-30], [1e30], [1e-44]], device="cuda")
    x[0, 9, 1], x[0, 10, 2], x[0, rows - 1, 0] = float("inf"), float("nan"), 1e6
    got = pkg.llmops.fc_Q4A(x, wq, N, nibble_signed=signed)
    want = torch.cat([pkg.llmops.fc_Q4A(part.contiguous(), wq, N, nibble_signed=signed) for part in x.split(60, dim=1)], dim=1)
    again = pkg.llmops.fc_Q4A(x, wq, N, nibble_signed=signed)
    assert torch.equal(got.view(torch.int32), again.view(torch.int32))  # fixed summation order
    assert torch.equal(got.isfinite(), want.isfinite()) and torch.equal(got.isnan(), want.isnan())
    got, want = got.nan_to_num(0, 0, 0), want.nan_to_num(0, 0, 0)
    # (the row of subnormal values: its results are a few units of the smallest number)
    assert ((got - want).abs() <= 2e-5 * want.abs().amax(-1, keepdim=True) + 1e-42).all()
    pkg.llmops.check_device_status()


def early_edges(graph):
    """Edges of a captured graph over which a kernel begins before the one in front of it has ended, and all of them."""
    cu, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t()
    g = ctypes.c_void_p(graph.raw_cuda_graph())
    assert cu.cuGraphGetEdges_v2(g, None, None, None, ctypes.byref(n)) == 0
    ends, data = [(ctypes.c_void_p * n.value)() for _ in range(2)], (ctypes.c_ubyte * (8 * n.value))()
    assert cu.cuGraphGetEdges_v2(g, ends[0], ends[1], data, ctypes.byref(n)) == 0
    return sum(data[8 * i + 2] == 1 for i in range(n.value)), n.value  # (bytes of an edge: from port, to port, type)


def test_quantizers_on_a_side_branch_do_not_begin_early(pkg):
    """Captured behind one another, or behind a kernel that something else follows already, quantizers are ordinary nodes; in
    one line with FCs they begin early.  The results are those of the eager calls."""
    ops, g = pkg.llmops, torch.Generator().manual_seed(9)
    K, N, dev = 512, 256, torch.device("cuda")
    w = ops.offline_FC_quant_Q4A((torch.randn(N, K, generator=g) * 0.02).cuda())
    xs = [torch.randn(1, 2, K, generator=g).cuda() for _ in range(4)]
    xq = [ops.QuantizedActivations(1, 2, K, 32, False, dev) for _ in xs]
    quantizers = [ops.QuantizeBatch([(x, q)]) for x, q in zip(xs, xq)]
    other = ops.QuantizeBatch([(xs[0], ops.QuantizedActivations(1, 2, K, 32, False, dev))])
    fcs = [ops.FCBatch([(q, w, N)]) for q in xq]
    want = [ops.fc_Q4A_q8(ops.quantize_activations(x, 32), w, N) for x in xs]
    main, side = torch.cuda.Stream(), torch.cuda.Stream()

    def line():
        for q, f in zip(quantizers, fcs):
            q.run(), f.run()

    def branch():
        start = torch.cuda.Event()
        start.record(main)
        side.wait_event(start)
        done = []
        with torch.cuda.stream(side):
            for q in quantizers:
                q.run()
                done.append(torch.cuda.Event())
                done[-1].record(side)
        for f, e in zip(fcs, done):
            main.wait_event(e)
            f.run()

    def row():
        for q in quantizers:
            q.run()

    def behind():  # the last quantizer behind an FC that another one follows already
        line()
        end = torch.cuda.Event()
        end.record(main)
        fcs[0].run()
        side.wait_event(end)
        with torch.cuda.stream(side):
            other.run()
            end.record(side)
        main.wait_event(end)

    torch.cuda.synchronize()
    for form, count in ((line, (7, 7)), (row, (0, 3)), (behind, (8, 9)), (branch, None)):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.stream(main):
            form()
            main.synchronize()
            with torch.cuda.graph(graph, stream=main):
                form()
        assert count is None or early_edges(graph) == count, form.__name__
        for f, q in zip(fcs, xq):
            f.outs[0].zero_(), q.buf.zero_()
        torch.cuda.synchronize()
        graph.replay()
        if form is row:
            [f.run() for f in fcs]
        torch.cuda.synchronize()
        assert all(torch.equal(f.outs[0], y) for f, y in zip(fcs, want)), form.__name__


def check_many_rows(pkg, oracle, fmt, rows, N, K, launches=None):
    g = torch.Generator().manual_seed(rows + N + K)
    W = torch.randn(N, K, generator=g) * 0.02
    x = torch.randn(1, rows, K, generator=g)
    if fmt == "q8c":
        wq, ws = oracle.restated.q8c_pack(W.numpy())
        want = oracle.restated.q8c_fc(x.numpy(), wq, ws, N)
        xd, wd, sd = x.cuda(), torch.from_numpy(wq).cuda(), torch.from_numpy(ws).cuda()
        run = lambda: pkg.c_ext.FC_evaluate_Q8C(xd, wd, sd, N)
    else:
        signed = isinstance(fmt, str)
        wq = oracle.restated.pack(W.numpy(), *((0, int(fmt[6:])) if signed else fmt))
        want = oracle.restated.fc(x.numpy(), wq, N, nibble_signed=signed)
        xd, wd = x.cuda(), torch.from_numpy(wq).cuda()
        run = lambda: pkg.llmops.fc_Q4A(xd, wd, N, nibble_signed=signed)
    got = run()
    assert torch.equal(got, run())  # fixed summation order
    if launches is not None:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            run()  # the stream's workspace
            stream.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                again = run()
        assert graph_nodes(graph) == launches
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, again)
    assert np.abs(got.cpu().numpy() - want).max() <= 2e-5 * np.abs(want).max()
    pkg.llmops.check_device_status()


@pytest.mark.parametrize("rows,N,K", [
    (8, 200, 520), (9, 200, 520), (16, 200, 520), (17, 200, 520), (32, 200, 520), (33, 200, 520),  # 1, 2 and 4 row tiles
    (16, 9500, 100), (17, 9500, 100),   # 297 stripes: two places on each of 148 SMs hold one CTA less
    (17, 9470, 100), (128, 1180, 250), (129, 1180, 250),  # as many CTAs as places; a row tile more
])
def test_q8c_row_tiles_and_the_line_to_the_gemm(pkg, oracle, rows, N, K):
    check_many_rows(pkg, oracle, "q8c", rows, N, K)


@pytest.mark.parametrize("K,sizes", [(1056, (300, 20, 200)), (2080, (200, 512, 20))])  # 200 and 512 rows: with a remainder
@pytest.mark.parametrize("fmt", ["q4", "q8c"])
def test_many_rows_captured_and_on_two_streams(pkg, fmt, K, sizes):
    """Calls with both tile sizes on one workspace, captured into a graph and replayed, and beside them eager calls on a
    second stream: all bit-equal to calls one by one (fixed summation orders)."""
    ops, N = pkg.llmops, 11008
    g = torch.Generator(device="cuda").manual_seed(4)
    W = torch.randn(N, K, generator=g, device="cuda") * 0.02
    if fmt == "q8c":
        w, s = pkg.c_ext.FC_quant_Q8C(W)
        fc = lambda x: ops.FC_evaluate_Q8C(x, w, s, N)
    else:
        w = ops.offline_FC_quant_Q4A(W)
        fc = lambda x: ops.fc_Q4A(x, w, N)
    inputs = [[torch.randn(1, rows, K, generator=g, device="cuda") for rows in sizes] for _ in range(3)]
    want = [[fc(x) for x in xs] for xs in inputs]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    static = [x.clone() for x in inputs[0]]
    with torch.cuda.stream(a):
        [fc(x) for x in static]  # the stream's workspace, at its largest
        a.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=a):
            outs = [fc(x) for x in static]
    for xs, ys in zip(inputs, want):
        with torch.cuda.stream(a):
            for t, x in zip(static, xs):
                t.copy_(x)
            graph.replay()
        with torch.cuda.stream(b):
            beside = [fc(x) for x in reversed(inputs[1])]
        torch.cuda.synchronize()
        assert all(torch.equal(o, y) for o, y in zip(outs, ys))
        assert all(torch.equal(o, y) for o, y in zip(beside, reversed(want[1])))


@pytest.mark.parametrize("rows,N,K", [
    (256, 11008, 4096),               # 128-row tiles, groups by 12
    (300, 9000, 2000),                # by 8, a last stage with three groups
    (129, 10000, 11008),
    (37, 11008, 4096),                # 64-row tiles, K divided by 3
    (512, 4096, 11008),               # undivided
    (17, 5000, 1000), (40, 2000, 4097),  # divided by 2 and 8
])
def test_q8c_many_rows_precision(pkg, rows, N, K):
    """The sums over K against 64 bits on the same codes and scales.  A rounding to nearest is off by 2.5e-8 of its sum in
    the root mean square; a chain of 12 groups holds 6.5 such errors of the whole sum's size (in squares), the second
    level, the division of K and the column scale four more at most: 8.1e-8.  One chain over K = 4096 gives 2.0e-7."""
    g = torch.Generator(device="cuda").manual_seed(rows + N + K)
    x = torch.randn(1, rows, K, generator=g, device="cuda")
    w, s = pkg.c_ext.FC_quant_Q8C(torch.randn(N, K, generator=g, device="cuda") * 0.02)
    codes, xs, _ = pkg.llmops.FC_dynamic_quantize_x(x[0], 32)
    Ng, Kg = w.shape[:2]
    q = w.view(Ng, Kg, 8, 32, 4).permute(0, 3, 1, 2, 4).reshape(Ng * 32, Kg * 32)[:N]
    want = (codes.double().view(rows, Kg, 32) * xs.double()[:, :, None]).view(rows, -1) @ q.double().t() * s[:N].double()
    got = pkg.c_ext.FC_evaluate_Q8C(x, w, s, N)[0].double()
    assert ((got - want).norm() / want.norm()).item() <= 8.1e-8


@pytest.mark.parametrize("rows", [40, 400])
def test_q8c_many_rows_beyond_the_finite_numbers(pkg, rows):
    """Sums that overflow, and inputs that are not finite, end as in the 8-row kernel.  (Finite rows: 2 x 40 roundings of
    2^-24, each of a part of the sum of the terms' sizes, about 16: 8e-5.)"""
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(1, rows, 1000, generator=g)
    x[0, 1], x[0, 2] = 1e38, -1e38
    x[0, 3, 700:], x[0, 5, 300], x[0, 6, 999], x[0, 7] = 3e38, float("inf"), float("nan"), float("nan")
    x = x.cuda()
    w, s = pkg.c_ext.FC_quant_Q8C((torch.rand(5000, 1000, generator=g) * 0.02 + 0.01).cuda())
    want = pkg.c_ext.FC_evaluate_Q8C(x[:, :8].contiguous(), w, s, 5000)
    got = pkg.c_ext.FC_evaluate_Q8C(x, w, s, 5000)[:, :8]
    assert torch.isinf(want[0, 1]).all() and torch.isinf(want[0, 2]).all() and torch.isinf(want[0, 3]).all()
    assert torch.allclose(got, want, rtol=0, atol=8e-5, equal_nan=True)


@pytest.mark.parametrize("qtype,G", [(0, 32), (1, 128)])
@pytest.mark.parametrize("K", [264, 260, 259])
@pytest.mark.parametrize("offset", [0, 4, 1])
def test_pack_load_widths(pkg, oracle, qtype, G, K, offset):
    """Rows that start on 32, 16 and 4 bytes take three widths of load: the same bytes."""
    g = torch.Generator().manual_seed(K + offset)
    W = torch.randn(33, K, generator=g) * 0.02
    store = torch.empty(33 * K + offset, device="cuda")
    w = store[offset:].view(33, K)
    w.copy_(W)
    got = pkg.llmops.offline_FC_quant_Q4A(w, qtype="q4_1" if qtype else "q4_0", group_k=G)
    assert np.array_equal(got.cpu().numpy(), oracle.restated.pack(W.numpy(), qtype, G))


@pytest.mark.parametrize("qtype,G", [(0, 32), (0, 128), (1, 32), (1, 128)])
@pytest.mark.parametrize("N,K", [(64, 512), (33, 520), (40, 516), (37, 515)])  # 32-, 16- and 4-byte loads; a column beyond N
def test_pack_scales_at_the_ends(pkg, oracle, qtype, G, N, K):
    """Groups on both sides of the scales between which the packer clamps nothing, in warps of ordinary ones; ties of the
    rounding (the values are multiples of half a step).  Bytes, so no tolerance."""
    g = torch.Generator().manual_seed(N * 7 + K + G)
    W = torch.randint(-14, 15, (N, K), generator=g).float() * 0.5
    # (where 1 / scale is infinite, what the reference's conversion to int makes of that is not defined)
    for row, scale in enumerate((2.0**-122, 2.0**-118, 2.0**-106, 2.0**-103, 2.0**-100, 2.0**-97, 2.0**97, 2.0**100, 2.0**103, 2.0**123)):
        W[row] *= scale
    W[10] = W[10].abs() + 1.0   # no zero among the extremes
    W[11, : K // 2] = 3.25      # equal values: scale 0 (Q4_1)
    want = oracle.restated.pack(W.numpy(), qtype, G)
    got = pkg.llmops.offline_FC_quant_Q4A(W.cuda(), qtype=("q4_0", "q4_1")[qtype], group_k=G).cpu().numpy()
    assert np.array_equal(got, want)


class EarlyWriter:
    """Rewrites a buffer with one of two contents by the embedding look-up, which lets its successor begin at once and then
    stores for as long as it takes: few CTAs, so that others find places beside them.  The values are whole numbers in fp32:
    bytes and halves of them are finite nibbles, codes and scales too."""

    def __init__(self, pkg, nbytes, ctas, seed):
        g, E = torch.Generator().manual_seed(seed), nbytes // 4 // ctas
        assert E * ctas * 4 == nbytes and E % 4 == 0
        self.table = torch.randint(-127, 128, (2 * ctas, E), generator=g).to(torch.int8).cuda()
        self.ids = torch.arange(2 * ctas).view(2, ctas).cuda()
        self.scales, self.out, self.pkg = torch.ones(2 * ctas, device="cuda"), torch.zeros(ctas, E, device="cuda"), pkg

    def __call__(self, k):
        self.pkg.llmops.embedding_q8c(self.out, self.ids[k], self.table, self.scales)


def alternating(step):
    """step(k, wait) twenty times for k = 0, 1, 0, ... without a wait or copy in between gives what it gives with waits (the same
    kernels on the same inputs: equal)."""
    step(1, True)
    want = [step(k, True) for k in (0, 1)]
    assert not torch.equal(want[0][-1], want[1][-1])
    got = [step(k % 2, False) for k in range(20)]
    torch.cuda.synchronize()
    for k in range(20):
        assert all(torch.equal(a, b) for a, b in zip(got[k], want[k % 2]))


EARLY_READERS = {  # what is written in front: its bytes, by how many CTAs, and who reads it
    **{f"weights, {rows} rows": (64 * 64 * 640, 16, lambda t, o, rows=rows: t.fc(t.x(rows, 2048), o.view(torch.int8).view(64, 64, 640), 2048))
       for rows in (1, 8, 20, 300)},
    **{f"activations, {rows} rows": (rows * 2048 * 4, 1 if rows < 4 else 4, lambda t, o, rows=rows: t.fc(o.view(1, rows, 2048), t.w, 2048))
       for rows in (1, 2, 8, 20, 300)},
    "activations, 129 rows and a remainder": (129 * 2080 * 4, 8, lambda t, o: t.fc(o.view(1, 129, 2080), t.wide, 9500)),
    **{f"int8 weights, {rows} rows": (64 * 64 * 1024, 16, lambda t, o, rows=rows: t.q8(t.x(rows, 2048), o.view(torch.int8).view(64, 64, 1024), t.s8))
       for rows in (1, 8, 300)},
    **{f"int8 scales, {rows} rows": (2048 * 4, 1, lambda t, o, rows=rows: t.q8(t.x(rows, 2048), t.w8, o.view(2048))) for rows in (1, 300)},
    **{f"int8 activations, {rows} rows": (rows * 2048 * 4, 1, lambda t, o, rows=rows: t.q8(o.view(1, rows, 2048), t.w8, t.s8))
       for rows in (1, 300)},
    "quantizer": (8 * 2048 * 4, 4, lambda t, o: t.ops.quantize_activations(o.view(1, 8, 2048), 32).codes()),
    "quantizer of its own": (20 * 2048 * 4, 4, lambda t, o: t.ops.FC_dynamic_quantize_x(o.view(20, 2048), 32)[0]),
    "table": (100 * 2048, 4, lambda t, o: t.look_up(o.view(torch.int8).view(100, 2048), t.s8[:100])),
    "table scales": (400, 1, lambda t, o: t.look_up(t.table, o.view(100))),
}


class EarlyInputs:
    def __init__(self, pkg):
        self.ops, self.q8c, self.g = pkg.llmops, pkg.c_ext, torch.Generator(device="cuda").manual_seed(2)
        r = lambda *s: torch.randn(*s, generator=self.g, device="cuda")
        self.w, self.wide = (self.ops.offline_FC_quant_Q4A(r(*s) * 0.02) for s in ((2048, 2048), (9500, 2080)))
        self.w8, self.s8 = pkg.c_ext.FC_quant_Q8C(r(2048, 2048) * 0.02)
        self.table = torch.randint(-127, 128, (100, 2048), generator=self.g, device="cuda").to(torch.int8)
        self.ids, self.kept = torch.arange(99, -1, -1, device="cuda"), {}
        self.wait = False
        self.fc = lambda x, w, N: self.done(self.ops.fc_Q4A(x, w, N))
        self.q8 = lambda x, w, s: self.done(pkg.c_ext.FC_evaluate_Q8C(x, w, s, 2048))

    def done(self, result):
        if self.wait:
            torch.cuda.synchronize()
        return result

    def x(self, rows, K):
        if (rows, K) not in self.kept:
            self.kept[rows, K] = torch.randn(1, rows, K, generator=self.g, device="cuda")
        return self.kept[rows, K]

    def look_up(self, table, scales):
        out = torch.empty(100, 2048, device="cuda")
        self.ops.embedding_q8c(out, self.ids, table, scales)
        return self.done(out)


@pytest.mark.parametrize("reader", EARLY_READERS)
def test_kernels_that_begin_early_wait_for_their_inputs(pkg, reader):
    """Weights, activations, scales and tables written by a kernel directly in front that releases its successor at once, again
    and again in the same buffer, which the reader of the time before may still read."""
    nbytes, ctas, read = EARLY_READERS[reader]
    t, write = EarlyInputs(pkg), EarlyWriter(pkg, nbytes, ctas, 5)
    t.x(1, 2048)

    def step(k, wait):
        t.wait = wait
        t.done(write(k))
        return [t.done(read(t, write.out))]

    alternating(step)


def test_kernels_that_begin_early_behind_one_another(pkg):
    """Chains of calls, each reading what the one in front computes, in memory that calls before them have used."""
    t, ops = EarlyInputs(pkg), pkg.llmops
    pack = lambda N, K: ops.offline_FC_quant_Q4A(torch.randn(N, K, generator=t.g, device="cuda") * 0.02)
    narrow = pack(64, 9500)
    xs = [{rows: torch.randn(1, rows, K, generator=t.g, device="cuda") for rows, K in ((1, 2048), (8, 2048), (20, 2048), (129, 2080))}
          for _ in range(2)]
    # ids from the quantizer: eight bytes each, the first of every group the 127 that makes the scale one
    ids = torch.randint(0, 127, (2, 8, 64, 4), generator=torch.Generator().manual_seed(1))
    ids[..., 0] = 127
    as_bytes = [ids[k].view(torch.int8).view(8, 2048).float().cuda() for k in (0, 1)]
    big = torch.randint(-127, 128, (128, 2048), generator=torch.Generator().manual_seed(1)).to(torch.int8).cuda()
    ones = torch.ones(128, device="cuda")

    ids_of = lambda k: t.done(ops.FC_dynamic_quantize_x(as_bytes[k], 32)[0]).view(torch.int64)
    codes = lambda x: t.done(ops.quantize_activations(x, 32)).codes()

    def look_up(i):
        out = torch.empty(*i.shape, 2048, device="cuda")
        ops.embedding_q8c(out, i, big, ones)
        return t.done(out)

    chains = [
        lambda k: t.fc(t.q8(t.fc(xs[k][8], t.w, 2048), t.w8, t.s8), t.w, 2048),
        lambda k: codes(t.fc(t.fc(xs[k][1], t.w, 2048), t.w, 2048)),
        lambda k: t.q8(t.fc(t.fc(xs[k][20], t.w, 2048), t.w, 2048), t.w8, t.s8),
        lambda k: t.fc(t.fc(xs[k][129], t.wide, 9500)[:, :8], narrow, 64),  # (129 rows: with a remainder)
        lambda k: t.fc(xs[k][129], t.wide, 9500),
        lambda k: t.fc(look_up(ids_of(k).view(-1)[:8]).view(1, 8, 2048), t.w, 2048),
        lambda k: look_up(ids_of(k)),
    ]

    def step(k, wait):
        t.wait = wait
        return [f(k) for f in chains]

    assert torch.equal(look_up(ids_of(0)), big[ids[0].view(8, 256).cuda()].float())
    alternating(step)
    pkg.llmops.check_device_status()


@pytest.mark.parametrize("reader", ["multi", "batch"])
@pytest.mark.parametrize("between", ["decode", "decode_quantizer", "prequantized", "prefill", "q8c", "quantizer", "look-up"])
def test_calls_without_the_flag_hold_a_flagged_successor_back(pkg, between, reader):
    """A kernel writes weights, a call without pdl=True follows, a call with it reads those weights, no copy or wait between:
    the same results as with waits (the same kernels on the same inputs: equal)."""
    ops, g = pkg.llmops, torch.Generator().manual_seed(3)
    K, N = 4096, 16384
    write = EarlyWriter(pkg, N // 32 * (K // 128) * 2176, 256, 1)
    w2 = write.out.view(torch.int8).view(N // 32, K // 128, 2176)
    x = torch.randn(1, 8, K, generator=g).cuda()
    x2 = ops.quantize_activations(torch.randn(1, 2, K, generator=g).cuda(), 128)
    w1 = ops.offline_FC_quant_Q4A((torch.randn(640, K, generator=g) * 0.02).cuda())
    w8, s8 = pkg.c_ext.FC_quant_Q8C((torch.randn(640, K, generator=g) * 0.02).cuda())
    x1, x32, w32 = ops.quantize_activations(x, 32), x.view(1, 32, K // 4), w1[:, :K // 128].contiguous()
    table, ids = pkg.ops.llmop_embedding_q8c(torch.randn(100, K, generator=g).cuda()), torch.arange(50).cuda()
    call = {"decode": lambda: ops.fc_Q4A(x[:, :1], w1, 640), "decode_quantizer": lambda: ops.fc_Q4A(x, w1, 640),
            "prequantized": lambda: ops.fc_Q4A_q8(x1, w1, 640), "prefill": lambda: ops.fc_Q4A(x32, w32, 640),
            "q8c": lambda: pkg.c_ext.FC_evaluate_Q8C(x, w8, s8, 640),
            "quantizer": lambda: ops.quantize_activations(x, 32).codes(), "look-up": lambda: table(ids)}[between]
    batch = ops.FCBatch([(x2, w2, N)], pdl=True)
    read = (lambda: ops.fc_Q4A_multi(x2, [w2], [N], pdl=True)[0]) if reader == "multi" else (lambda: batch.run()[0].clone())

    def step(k, wait):
        out = []
        for f in (lambda: write(k), call, read):
            out.append(f())
            if wait:
                torch.cuda.synchronize()
        return out[1:]

    alternating(step)
