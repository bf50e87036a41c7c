"""Edges of the ranges that the kernels' tiles and dispatch rules draw: remainders, the smallest and the largest sizes."""
import pytest
import torch

import e3nn_b200
from conftest import rel_err
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
    src, dst, shift, rowptr = e3nn_b200.nn.neighbor_list_pbc(pos.to(DEV), box, 5.0)
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
