"""Edges of the ranges that the kernels' tiles and dispatch rules draw: remainders, the smallest and the largest sizes."""
import pytest
import torch

import e3nn_b200
from conftest import fp32_bound, rel_err
from e3nn_b200 import layouts
from e3nn_b200 import nn as bnn
from e3nn_b200 import o3
from oracle import e3nn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


# ----------------------------------------------------------------------------- CSR: 2,048-key blocks, 8-bit digits
@pytest.mark.parametrize("E,N", [(1, 2), (31, 256), (2047, 257), (2048, 65536), (2049, 65537), (100_001, 2), (600_000, 1_000_003)])
def test_csr_block_and_digit_edges(E, N):
    g = torch.Generator().manual_seed(E)
    dst = torch.randint(0, N, (E,), generator=g)
    dst[-1] = N - 1
    perm, rowptr = e3nn_b200.csr_from_dst(dst.to(DEV), N)
    ref_perm, ref_rowptr = orc.csr_from_dst(dst, N)
    assert torch.equal(perm.cpu(), ref_perm) and torch.equal(rowptr.cpu(), ref_rowptr)


# ----------------------------------------------------------------------------- neighbour list: a row in shared memory or not
@pytest.mark.parametrize("extra", [250, 270, 600])
def test_neighbor_list_dense_rows(extra):
    """`extra` atoms inside one ball of radius 2 (rows of about that many entries: around and above the 256 that are
    ranked in shared memory) plus a thin gas, against all pairs on the host."""
    g = torch.Generator().manual_seed(extra)
    box, n_gas = 20.0, 37
    ball = torch.nn.functional.normalize(torch.randn(extra, 3, generator=g), dim=-1) * 2.0 * torch.rand(extra, 1, generator=g) ** (1 / 3)
    pos = torch.cat([ball + 0.5, torch.rand(n_gas, 3, generator=g) * box])      # the ball lies across the corner of the box
    src, dst, shift, rowptr = bnn.neighbor_list_pbc(pos.to(DEV), box, 5.0)
    p = pos.double() - torch.floor(pos.double() / box) * box
    d = p[None, :, :] - p[:, None, :]
    d = d - box * torch.round(d / box)
    near = d.pow(2).sum(-1) <= 25.0
    near.fill_diagonal_(False)
    ref_dst, ref_src = near.nonzero(as_tuple=True)
    assert int(near.sum(1).max()) >= extra - 1
    assert torch.equal(dst.cpu(), ref_dst) and torch.equal(src.cpu(), ref_src)
    vec = pos.to(DEV)[src] - pos.to(DEV)[dst] + shift
    # coordinates of up to 20 in fp32: three roundings of 2^-24 * 20
    assert (vec.cpu().double() - d[ref_dst, ref_src]).abs().max().item() < 4e-6
    assert int(rowptr[-1]) == src.numel()


# ----------------------------------------------------------------------------- fp32 contractions on register tiles
TILE_LAYOUTS = [
    ("1x0e+33x1o", "0e+2x1o", "17x0e+3x1o+16x1e"),                 # one channel, a chunk of 32 + 1, two second-operand channels
    ("65x0e+5x1o+2x2e", "1x0e+1x1o+1x2e", "130x0e+64x1o+1x2e"),    # column blocks of 128 + 2, one output channel
    ("4x3o+7x2e", "3o+2e+1o", "9x0e+33x3o+2x1o"),                  # l = 3 throughout
    ("3x4e+2x0e", "2x1o+4e", "5x4e+2x0e+3x3o"),                    # l = 4: staged without the unrolled irreps, derived products backward
    ("2x0e+3x1o", "33x0e+9x1o+40x2e", "9x0e+33x1o+5x2e"),          # operands exchanged: the second one's channels are taken by 32
    ("9x0e+8x1o", "5x0e+12x1o", "8x0e+8x1o"),                      # around eight channels a chunk
    ("2x0e+1x1o", "3x0e+1x1o", "40x0e+7x1o"),                      # a few channels: the table-driven kernel forward
    ("1x0e+2x2e", "20x0e+20x4e", "5x0e+6x2e"),                     # l = 4 in the wide operand, which stays second
    ("8x0e+8x1o", "5x0e", "8x0e+8x1o+4x2e"),                       # scalar second operand, an output no path writes
]


@pytest.mark.parametrize("rows", [1, 31, 129, 1000])
@pytest.mark.parametrize("layout", TILE_LAYOUTS)
def test_fp32_product_tiles(layout, rows):
    """Forward and all gradients; bound: 1e-5 x RMS, the fp32 parity bound of this path."""
    g = torch.Generator().manual_seed(rows)
    tp = o3.FullyConnectedTensorProduct(*layout)
    x = torch.randn(rows, tp.irreps_in1.dim, generator=g)
    y = torch.randn(rows, tp.irreps_in2.dim, generator=g)
    go = torch.randn(rows, tp.irreps_out.dim, generator=g)
    ins = [(i.i_in1, i.i_in2, i.i_out, i.connection_mode, i.has_weight) for i in tp.instructions]
    x64, y64, w64 = (t.detach().double().requires_grad_(True) for t in (x, y, tp.weight))
    ref = orc.tensor_product(*(str(i) for i in (tp.irreps_in1, tp.irreps_in2, tp.irreps_out)), ins, x64, y64, w64, True)
    ref_g = torch.autograd.grad(ref, [x64, y64, w64], go.double())
    tp = tp.to(DEV)
    xd, yd = x.to(DEV).requires_grad_(True), y.to(DEV).requires_grad_(True)
    out = tp(xd, yd)
    got_g = torch.autograd.grad(out, [xd, yd, tp.weight], go.to(DEV))
    assert rel_err(out.detach().cpu(), ref.detach()) < 1e-5
    for got, want in zip(got_g, ref_g):
        assert rel_err(got.cpu(), want) < 1e-5
    # each operand gradient on its own takes another instance of the kernel
    for n, leaf in enumerate((xd, yd)):
        other = tp(xd if n == 0 else xd.detach(), yd if n == 1 else yd.detach(), tp.weight.detach())
        assert rel_err(torch.autograd.grad(other, leaf, go.to(DEV))[0].cpu(), ref_g[n]) < 1e-5


@pytest.mark.parametrize("rows", [500, 4000])
@pytest.mark.parametrize("layout", [("4x0e+4x1o", "4x0e+4x1o", "5x0e+3x1o"), ("9x0e+5x1o", "9x0e+9x1o", "70x0e+130x1o"), ("16x0e+4x2e", "16x0e+4x2e", "9x0e+2x2e")])
def test_fp32_product_weight_gradient_over_pairs(layout, rows):
    """Poorly filled chunks: at the larger row counts the weight gradient contracts pairs of channels.  Bound: 1e-5 x RMS, the
    fp32 parity bound of this path."""
    g = torch.Generator().manual_seed(rows)
    tp = o3.FullyConnectedTensorProduct(*layout)
    x, y, go = (torch.randn(rows, d, generator=g) for d in (tp.irreps_in1.dim, tp.irreps_in2.dim, tp.irreps_out.dim))
    ins = [(i.i_in1, i.i_in2, i.i_out, i.connection_mode, i.has_weight) for i in tp.instructions]
    w64 = tp.weight.detach().double().requires_grad_(True)
    ref = orc.tensor_product(*(str(i) for i in (tp.irreps_in1, tp.irreps_in2, tp.irreps_out)), ins, x.double(), y.double(), w64, True)
    (want,) = torch.autograd.grad(ref, w64, go.double())
    tp = tp.to(DEV)
    (got,) = torch.autograd.grad(tp(x.to(DEV), y.to(DEV)), tp.weight, go.to(DEV))
    assert rel_err(got.cpu(), want) < 1e-5


@pytest.mark.parametrize("layout,rows", [(("65x0e+33x1o+32x2e", "1x0e+1x1o+1x2e", "32x0e+32x1o+32x2e"), 4000),      # 6 blocks of channels
                                         (("320x0e+64x1o", "300x0e+60x1o", "2x0e"), 6000),                      # 12, rows in two turns
                                         (("3x0e+2x1o", "40x0e+70x1o", "8x0e+4x1o"), 1000),                     # operands exchanged, 5
                                         (("32x0e", "1x0e+1x1o", "8x0e+8x1o"), 100)])                           # one: no partials
def test_fp32_product_second_operand_gradient_repeats(layout, rows):
    """Bit for bit: the same on every call, and for a row whatever rows stand beside it."""
    g = torch.Generator().manual_seed(rows)
    tp = o3.FullyConnectedTensorProduct(*layout).to(DEV)
    x, y, go = (torch.randn(rows, d, generator=g).to(DEV) for d in (tp.irreps_in1.dim, tp.irreps_in2.dim, tp.irreps_out.dim))

    def grad(sl):
        leaf = y[sl].clone().requires_grad_(True)
        return torch.autograd.grad(tp(x[sl], leaf), leaf, go[sl])[0]

    first = grad(slice(None))
    assert torch.equal(grad(slice(rows - 70, None)), first[rows - 70 :])
    for _ in range(5):
        assert torch.equal(grad(slice(None)), first)


@pytest.mark.parametrize("tail", ["2x3o", "2x0e"])
def test_fp32_product_many_outputs_wide_second_operand(tail):
    """33 output irreps (32 go out in one launch) and operands of 1,280 columns: with the l = 3 irrep last, the first 32
    fit a block's shared memory and the last does not.  Outputs start from NaN.  Bound: 1e-5 x RMS, or 1.5 times the distance of
    plain fp32 arithmetic on the host where that is larger (sums of thousands of terms)."""
    rows = 12
    g = torch.Generator().manual_seed(5)
    outs = "+".join(["2x0e"] * 32 + [tail])
    ins = [(i, j, k, "uvw", True) for k, l in enumerate([0] * 32 + [3 if tail == "2x3o" else 0])
           for i, j in [(0, 0), (3, 3), (0, 3), (3, 0)] if (l == 3) == (i != j)]
    tp = o3.TensorProduct("80x0e+80x1o+80x2e+80x3o", "80x0e+80x1o+80x2e+80x3o", outs, ins)
    x, y = torch.randn(rows, tp.irreps_in1.dim, generator=g), torch.randn(rows, tp.irreps_in2.dim, generator=g)
    go = torch.randn(rows, tp.irreps_out.dim, generator=g)
    want = []
    for dtype in (torch.float64, torch.float32):
        leaves = [t.detach().to(dtype).requires_grad_(True) for t in (x, y, tp.weight)]
        ref = orc.tensor_product(*(str(i) for i in (tp.irreps_in1, tp.irreps_in2, tp.irreps_out)), ins, *leaves, True)
        want.append([ref.detach()] + list(torch.autograd.grad(ref, leaves, go.to(dtype))))
    tp = tp.to(DEV)
    xd, yd = x.to(DEV).requires_grad_(True), y.to(DEV).requires_grad_(True)
    out = torch.full((rows, tp.irreps_out.dim), float("nan"), device=DEV)
    with torch.no_grad():
        tp._uvw_run(xd, yd, tp.weight, out, False)
    got = [out] + list(torch.autograd.grad(tp(xd, yd), [xd, yd, tp.weight], go.to(DEV)))
    for a, r64, r32 in zip(got, *want):
        assert rel_err(a.cpu(), r64) < fp32_bound(rel_err(r32, r64))


def test_fp32_rounding_of_long_sums_over_narrow_blocks():
    """Thousands of terms from operand blocks of one and two channels, summed 32 at a time as with wide blocks.  Bound on the
    2-norm: 1.5 times, in quadrature, three roundings of 2^-24 and the random walks of a run of 32 and of the K / 32 runs, 0.3 x
    2^-24 x sqrt(n) each (0.3: the mean rounding error of a sum that grows to its last size).  One walk of K steps: 9e-7."""
    g = torch.Generator().manual_seed(0)
    tp = o3.FullyConnectedTensorProduct("+".join(["2x0e"] * 33), "80x0e", "4x0e")
    lin = o3.Linear("+".join(["1x0e"] * 3000), "32x0e")
    x, y, z = (torch.randn(100, d, generator=g) for d in (tp.irreps_in1.dim, tp.irreps_in2.dim, lin.irreps_in.dim))
    ins = [(i.i_in1, i.i_in2, i.i_out, i.connection_mode, i.has_weight) for i in tp.instructions]
    ref = orc.tensor_product(*(str(i) for i in (tp.irreps_in1, tp.irreps_in2, tp.irreps_out)), ins, x.double(), y.double(),
                             tp.weight.detach().double(), True)
    ref_lin = orc.linear(str(lin.irreps_in), str(lin.irreps_out), z.double(), lin.weight.detach().double())
    with torch.no_grad():
        for got, want, k in ((tp.to(DEV)(x.to(DEV), y.to(DEV)), ref, 5280), (lin.to(DEV)(z.to(DEV)), ref_lin, 3000)):
            err = ((got.cpu().double() - want).norm() / want.norm()).item()
            assert err < 1.5 * 2.0**-24 * (9 + 0.09 * (32 + k / 32)) ** 0.5, (k, err)


@pytest.mark.parametrize("rows", [1, 257])
@pytest.mark.parametrize("irreps", [("1x0e+40x1o+3x2e", "200x0e+2x0e+17x1o"), ("70x0e+9x4e", "9x4e+16x0e+5x1o"), ("64x0e+64x3o", "32x0e+64x3o"),
                                    ("40x16e+3x31o+2x0e", "70x16e+130x31o+5x0e"),
                                    ("+".join(["1x0e", "2x1o"] * 24), "7x0e+5x1o"), ("+".join(["1x0e", "2x1o"] * 25), "7x0e+5x1o+1x0o")])
def test_fp32_linear_tiles(irreps, rows):
    """Forward, transposed (two outputs of different width from one input, an input nothing reads) and weight gradient; one
    layout has more components than a tile of 128 columns has rows, up to the largest irrep taken, two have many narrow blocks."""
    g = torch.Generator().manual_seed(rows)
    lin = o3.Linear(*irreps)
    x, go = torch.randn(rows, lin.irreps_in.dim, generator=g), torch.randn(rows, lin.irreps_out.dim, generator=g)
    x64, w64 = x.double().requires_grad_(True), lin.weight.detach().double().requires_grad_(True)
    ref = orc.linear(irreps[0], irreps[1], x64, w64)
    ref_g = torch.autograd.grad(ref, [x64, w64], go.double())
    lin, xd = lin.to(DEV), x.to(DEV).requires_grad_(True)
    out = lin(xd)
    got_g = torch.autograd.grad(out, [xd, lin.weight], go.to(DEV))
    assert rel_err(out.detach().cpu(), ref.detach()) < 1e-5
    for got, want in zip(got_g, ref_g):
        assert rel_err(got.cpu(), want) < 1e-5


# ----------------------------------------------------------------------------- pipelined convolution on permuted edges
@pytest.mark.parametrize("layout", ["cfg3_11", "cfg5_23"])
@pytest.mark.parametrize("nodes,edges", [(1, 1), (3, 33), (200, 64), (40, 1500), (1500, 6001)])
def test_conv_pipelined_permuted_edges(layout, nodes, edges):
    """Batches of 32 slots, rows longer than a batch, empty rows, fewer rows than SMs; the permuted call must give what the
    sorted one gives (same kernels, same order within a row) and agree with the direct-load kernels."""
    g = torch.Generator().manual_seed(edges)
    tp = layouts.bench_conv_tp(layout)
    dst = torch.randint(0, nodes, (edges,), generator=g)
    src = torch.randint(0, nodes, (edges,), generator=g)
    perm, rowptr = e3nn_b200.csr_from_dst(dst.to(DEV), nodes)
    x, vec, w = torch.randn(nodes, tp.irreps_in1.dim, generator=g), torch.randn(edges, 3, generator=g), torch.randn(edges, tp.weight_numel, generator=g)
    go = torch.randn(nodes, tp.irreps_out.dim, generator=g).to(DEV)

    def call(order, perm_arg):
        xd, vd, wd = (t.to(DEV).requires_grad_(True) for t in (x, vec[order], w[order]))
        out = e3nn_b200.conv_uvu(tp, xd, vd, src[order].to(DEV), rowptr, wd, perm=perm_arg, scale=0.5, edge_attr_is_vector=True,
                                 check_indices=True)
        return [out.detach()] + list(torch.autograd.grad(out, [xd, vd, wd], go))

    p = perm.cpu()
    permuted, in_order = call(torch.arange(edges), perm), call(p, None)
    assert torch.equal(permuted[0], in_order[0])
    assert torch.equal(permuted[2][perm], in_order[2]) and torch.equal(permuted[3][perm], in_order[3])
    lib = tp._uvu_module().lib
    lib.e3b_conv_select(1)
    try:
        direct = call(torch.arange(edges), perm)
    finally:
        lib.e3b_conv_select(0)
    # two fp32 summation orders of rows of up to 60 messages; 2e-5 x RMS as for the sorted form of these kernels
    for a, b in zip(permuted, direct):
        assert rel_err(a.cpu(), b.cpu().double()) < 2e-5


@pytest.mark.parametrize("layout", ["cfg3_11", "cfg5_23"])
@pytest.mark.parametrize("bad", ["source", "perm", "perm_negative"])
def test_conv_pipelined_skips_a_bad_index(layout, bad):
    """One slot with a source or a permutation entry out of range: reported, and every other edge and row is what it is without
    that edge, bit for bit (its weights set to zero give the same sums).  Bound for the node-feature gradient, whose atomics
    come in any order: two sums of about 30 edges, a rounding of 2^-24 each (twice that for rows of twice the edges)."""
    g = torch.Generator().manual_seed(3)
    tp, nodes, edges, slot = layouts.bench_conv_tp(layout), 50, 1500, 777
    dst, src = torch.randint(0, nodes, (edges,), generator=g), torch.randint(0, nodes, (edges,), generator=g).to(DEV)
    perm, rowptr = e3nn_b200.csr_from_dst(dst.to(DEV), nodes)
    lost = int(perm[slot])
    assert lost != 0
    x, vec, w = (torch.randn(*s, generator=g).to(DEV) for s in ((nodes, tp.irreps_in1.dim), (edges, 3), (edges, tp.weight_numel)))
    go = torch.randn(nodes, tp.irreps_out.dim, generator=g).to(DEV)

    def call(src, perm, w):
        leaves = [t.clone().requires_grad_(True) for t in (x, vec, w)]
        out = e3nn_b200.conv_uvu(tp, leaves[0], leaves[1], src, rowptr, leaves[2], perm=perm, scale=0.5, edge_attr_is_vector=True)
        return [out.detach()] + list(torch.autograd.grad(out, leaves, go))

    w_without = w.clone()
    w_without[lost] = 0.0
    want = call(src, perm, w_without)
    e3nn_b200.check_status()
    bad_src, bad_perm = src.clone(), perm.clone()
    if bad == "source":
        bad_src[lost] = nodes
    else:
        bad_perm[slot] = edges if bad == "perm" else -1
    from e3nn_b200 import _lib

    poll, _lib.poll_status = _lib.poll_status, lambda *a: None      # (the report of the forward pass would be raised in the backward)
    try:
        got = call(bad_src, bad_perm, w)
    finally:
        _lib.poll_status = poll
    with pytest.raises(IndexError):
        e3nn_b200.check_status()
    rest = torch.arange(edges, device=DEV) != lost
    assert torch.equal(got[0], want[0])
    assert torch.equal(got[2][rest], want[2][rest]) and torch.equal(got[3][rest], want[3][rest])
    assert rel_err(got[1].cpu(), want[1].cpu().double()) < 2 * 2 * 30 * 2.0**-24


# ----------------------------------------------------------------------------- edge embedding: gradient of its weights
@pytest.mark.parametrize("edges", [1, 33, 4001])
@pytest.mark.parametrize("act,hidden,nb,with_pos", [("silu", 64, 8, False), ("tanh", 32, 5, True), ("relu", 128, 16, True), ("silu", 96, 9, False)])
def test_edge_embed_weight_gradient(act, hidden, nb, with_pos, edges):
    """Against the same chain in fp64; 1e-5 x RMS, the fp32 parity bound of this path."""
    g = torch.Generator().manual_seed(edges + nb)
    N, c = 50, 5.0
    pos = torch.rand(N, 3, generator=g) * 6.0
    src = torch.randint(0, N, (edges,), generator=g)
    dst = (src + 1 + torch.randint(0, N - 1, (edges,), generator=g)) % N
    w0, gh = torch.randn(nb, hidden, generator=g), torch.randn(edges, hidden, generator=g)
    w_scale, act_scale = nb ** -0.5, bnn.normalize2mom_constant(act)
    f = {"silu": torch.nn.functional.silu, "tanh": torch.tanh, "relu": torch.relu}[act]
    p64, w64 = pos.double().requires_grad_(True), w0.double().requires_grad_(True)
    h64 = act_scale * f(bnn.bessel((p64[src] - p64[dst]).norm(dim=-1), nb, c) @ (w64 * w_scale))
    ref = torch.autograd.grad(h64, [p64, w64], gh.double())

    pd, wd = pos.to(DEV).requires_grad_(with_pos), w0.to(DEV).requires_grad_(True)

    def embed(weight_grad):
        return bnn.edge_embed(pd, src.to(DEV), dst.to(DEV), None, wd, c, w_scale, act_scale, act, check_indices=True, weight_grad=weight_grad)

    vec, h = embed(True)
    assert vec.requires_grad == with_pos
    got = torch.autograd.grad(h, ([pd] if with_pos else []) + [wd], gh.to(DEV))
    assert rel_err(got[-1].cpu(), ref[1]) < 1e-5
    if with_pos:
        assert rel_err(got[0].cpu(), ref[0]) < 1e-5
    again = torch.autograd.grad(embed(True)[1], wd, gh.to(DEV))[0]
    assert torch.equal(again, got[-1])           # fixed summation order
    with pytest.raises(NotImplementedError):
        torch.autograd.grad(embed(False)[1], wd, gh.to(DEV))


# ----------------------------------------------------------------------------- weight gradient of a dense layer
@pytest.mark.parametrize("rows,m,n,offset", [(1, 32, 16, 0), (63, 64, 144, 0), (1025, 96, 1472, 0), (20_011, 64, 128, 1), (777, 33, 130, 0)])
def test_dense_layer_weight_gradient(rows, m, n, offset):
    """64 x 128 tiles, stages of 16 rows, splits; `offset` floats in front of the operands (no 16-byte loads).  Bound: the random
    walk of the roundings of runs of at most 2,048 rows, 2^-24 sqrt(rows of a run), relative to the sums' size."""
    from e3nn_b200 import _lib

    g = torch.Generator().manual_seed(rows)
    x, go = torch.randn(rows, m, generator=g), torch.randn(rows, n, generator=g)
    ref = 0.5 * (x.double().t() @ go.double())
    xd, gd = torch.empty(offset + rows * m, device=DEV), torch.empty(offset + rows * n, device=DEV)
    xd[offset:], gd[offset:] = x.to(DEV).view(-1), go.to(DEV).view(-1)
    core, out = _lib.core(), torch.empty(m, n, device=DEV)
    need = core.e3b_matmul_tn_scratch_bytes(rows, m, n)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device=DEV)
    args = (_lib._ptr(xd[offset:]), _lib._ptr(gd[offset:]), rows, m, n, 0.5, _lib._ptr(out), _lib._ptr(scratch))
    assert core.e3b_matmul_tn(*args, need, _lib.stream_ptr()) == 0
    err = (out.cpu().double() - ref).norm() / ref.norm()
    assert err < 2.0**-24 * (4 + min(rows, 2048) ** 0.5), err
    first = out.clone()
    assert core.e3b_matmul_tn(*args, need, _lib.stream_ptr()) == 0 and torch.equal(out, first)
    if need > 0:
        assert core.e3b_matmul_tn(*args, need - 1, _lib.stream_ptr()) == -1


def test_dense_layer_weight_gradient_past_eight_waves():
    """Blocks of 16,384 rows, summed 2,048 at a time.  Bound: twice the random walk of such a run's roundings, 0.3 x 2^-24 x
    sqrt(2048) of the sums' size (0.3: the mean rounding error of a sum that grows to its last size)."""
    from e3nn_b200 import _lib

    rows, m, n = 131_072, 2048, 2048
    g = torch.Generator(device=DEV).manual_seed(1)
    x, go = torch.randn(rows, m, generator=g, device=DEV), torch.randn(rows, n, generator=g, device=DEV)
    core, out = _lib.core(), torch.empty(m, n, device=DEV)
    scratch = torch.empty(core.e3b_matmul_tn_scratch_bytes(rows, m, n), dtype=torch.uint8, device=DEV)
    assert scratch.numel() == 8 * m * n * 4
    assert core.e3b_matmul_tn(_lib._ptr(x), _lib._ptr(go), rows, m, n, 0.5, _lib._ptr(out), _lib._ptr(scratch), scratch.numel(),
                              _lib.stream_ptr()) == 0
    ref = torch.zeros(m, n, dtype=torch.float64, device=DEV)
    for z in range(0, rows, 16_384):
        ref += 0.5 * (x[z : z + 16_384].double().t() @ go[z : z + 16_384].double())
    err = ((out.double() - ref).norm() / ref.norm()).item()
    assert err < 2.0**-24 * (4 + 0.6 * 2048**0.5), err


# ----------------------------------------------------------------------------- dense layers on tensor cores
@pytest.mark.parametrize("rows", [1, 33, 127, 1000])
@pytest.mark.parametrize("width", [96, 1472])
def test_dense_layer_tiles(width, rows):
    """128-row tiles whose output leaves in boxes of 32 x 32: the last box ends with the rows.  The output lies between guard
    rows that must keep their values.  Bound: 4e-5 x RMS, the split-operand bound of this path."""
    from e3nn_b200 import _lib

    g = torch.Generator().manual_seed(rows)
    layer = bnn.FullyConnectedNet([64, width], math_mode="tf32x3").layer0
    w = torch.randn(64, width, generator=g)
    for transpose, gs in enumerate(layer._tc_specs()):
        a, b = (w, layer._scale()) if not transpose else (w.t(), layer._scale())
        x = torch.randn(rows, a.shape[0], generator=g)
        buf = torch.full((rows + 2, a.shape[1]), 7.0, device=DEV)
        _lib.tc_gemm_module(gs).run(x.to(DEV), None, w.to(DEV), buf[1 : rows + 1], 2)
        e3nn_b200.check_status()
        assert torch.all(buf[0] == 7.0) and torch.all(buf[-1] == 7.0)
        assert rel_err(buf[1 : rows + 1].cpu(), b * (x.double() @ a.double())) < 4e-5


# ----------------------------------------------------------------------------- Gate by channels
@pytest.mark.parametrize("rows", [1, 2, 333])
@pytest.mark.parametrize("scalars,gates,gated", [("5x0e", "3x0e+2x0e+4x0e+1x0e", "3x1o+2x2e+4x3o+1x4e"), ("", "70x0e", "70x1o"), ("300x0e", "", "")])
def test_gate_channels(scalars, gates, gated, rows):
    """One to nine components a channel, more channels than a block has threads, gates only, scalars only; the gradient by
    channels against the one by columns (the same formula: differences of the last bit) and the forward against fp64."""
    from e3nn_b200 import _lib

    silu, sig = torch.nn.functional.silu, torch.sigmoid
    gate = bnn.Gate(scalars, [silu] * len(o3.Irreps(scalars)), gates, [sig] * len(o3.Irreps(gates)), gated).to(DEV)
    assert gate._ch_covers
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, gate.irreps_in.dim, generator=g).to(DEV).requires_grad_(True)
    go = torch.randn(rows, gate.irreps_out.dim, generator=g).to(DEV)
    out = gate(x)
    (got,) = torch.autograd.grad(out, x, go)
    by_columns = torch.empty_like(x)
    rc = _lib.core().e3b_gate_bwd(_lib._ptr(x), _lib._ptr(go), _lib._ptr(gate._in_tbl), _lib._ptr(gate._in_cst), _lib._ptr(by_columns), rows,
                                  x.shape[1], go.shape[1], _lib.stream_ptr())
    assert rc == 0
    assert rel_err(got.cpu(), by_columns.cpu().double()) < 1e-6
    t, c, x64 = gate._out_tbl.cpu().long(), gate._out_cst.cpu().double(), x.detach().cpu().double()
    f = lambda act, v: torch.where(act == 0, silu(v), torch.sigmoid(v))      # noqa: E731
    ref = torch.where(t[:, 1] < 0, c * f(t[:, 2], x64[:, t[:, 0]]), x64[:, t[:, 0]] * c * f(t[:, 2], x64[:, t[:, 1].clamp_min(0)]))
    assert rel_err(out.detach().cpu(), ref) < 1e-5


# ----------------------------------------------------------------------------- Gate as the Linear's epilogue: gated scalars
GATED_SCALARS = [
    # gate arguments, the Linear's output irreps, whether every gate stands in an irrep before the scalars it gates
    (("16x0e", ["silu"], "8x0o", ["tanh"], "8x0e"), "8x0o+24x0e", True),
    (("16x0e", ["silu"], "8x0e+4x0e", ["sigmoid", "tanh"], "8x0e+4x1o"), "16x0e+12x0e+8x0e+4x1o", True),
    (("16x0e", ["silu"], "8x0e", ["sigmoid"], "8x0e"), "32x0e", False),
    (("16x0e", ["silu"], "8x0e", ["sigmoid"], "8x0o"), "8x0o+24x0e", False),
]


@pytest.mark.parametrize("rows", [1, 5000])
@pytest.mark.parametrize("args,irreps,ordered", GATED_SCALARS)
def test_linear_gate_gated_scalars(args, irreps, ordered, rows):
    """The module against the fp64 oracle; where the gates' irreps come first, the fused entry point too, from gate slots that
    held NaN.  1e-5 x RMS, the fp32 parity bound of this path."""
    from e3nn_b200 import _lib

    f = {"silu": torch.nn.functional.silu, "tanh": torch.tanh, "sigmoid": torch.sigmoid}
    gate = bnn.Gate(args[0], [f[a] for a in args[1]], args[2], [f[a] for a in args[3]], args[4])
    lin = o3.Linear("24x0e+12x0o+8x1o", irreps)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, lin.irreps_in.dim, generator=g)
    ref = orc.gate(*args, orc.linear(str(lin.irreps_in), str(lin.irreps_out), x.double(), lin.weight.detach().double()))
    pair = bnn.LinearGate(lin, gate, fuse=True).to(DEV)
    xd = x.to(DEV)
    with torch.no_grad():
        assert rel_err(pair(xd).cpu(), ref) < 1e-5
    if ordered:
        gates = torch.full((rows, pair.n_slots), float("nan"), device=DEV)
        out = torch.full((rows, gate.irreps_out.dim), float("nan"), device=DEV)
        rc = _lib.core().e3b_dense_fwd_gate(lin._plan_host.ctypes.data, _lib._ptr(lin._plan_on(xd.device, False)), _lib._ptr(xd),
                                            _lib._ptr(lin.weight.detach()), _lib._ptr(pair._fuse_tbl), _lib._ptr(pair._fuse_cst),
                                            _lib._ptr(gates), pair.n_slots, _lib._ptr(out), out.shape[1], rows, _lib.stream_ptr())
        assert rc == 0
        assert rel_err(out.cpu(), ref) < 1e-5
