"""Host logic of the weight-shared paths, checked on the CPU: the dense plans, interpreted here in numpy as the kernels read
them (the first part: per-row weights and the Gate epilogue above l = 3; the second part: everything else), and the
construction of the transposed products that give the operand gradients."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from e3nn_b200 import o3
from e3nn_b200.o3._dense_plan import MAGIC, linear_plan
from oracle import e3nn_oracle as orc


def _i2f(v: int) -> float:
    return float(np.int32(v).view(np.float32))


def run_plan(plan: np.ndarray, x1: np.ndarray, x2, W: np.ndarray, accumulate_into=None) -> np.ndarray:
    """out[z, out_off + w * dim3 + k] (+)= sum_K A[z, k, K] * W[wbase(K) + w * wstride], A from the CG triples."""
    assert plan[0] in (MAGIC, 0x65336250)
    d1, d2, dout, n_groups = (int(v) for v in plan[1:5])
    off_groups, off_kent, off_pathk, off_cg = (int(v) for v in plan[7:11])
    assert x1.shape[1] == d1 and (x2 is None or x2.shape[1] == d2)
    Z = x1.shape[0]
    out = np.zeros((Z, dout)) if accumulate_into is None else accumulate_into
    for g in range(n_groups):
        out_off, mul_out, dim3, K, kent_start, w_stride = (int(v) for v in plan[off_groups + 6 * g : off_groups + 6 * g + 6])
        block = np.zeros((Z, mul_out, dim3))
        for kk in range(K):
            path, x1off, x2off, wbase = (int(v) for v in plan[off_kent + 4 * (kent_start + kk) : off_kent + 4 * (kent_start + kk) + 4])
            wrow = W[wbase + np.arange(mul_out) * w_stride]
            for k in range(dim3):
                pk = int(plan[off_pathk + path]) + 2 * k
                cstart, ccount = int(plan[pk]), int(plan[pk + 1])
                a = np.zeros(Z)
                for c in range(cstart, cstart + ccount):
                    i, j, coef = int(plan[off_cg + 3 * c]), int(plan[off_cg + 3 * c + 1]), _i2f(plan[off_cg + 3 * c + 2])
                    a += coef * x1[:, x1off + i] * (x2[:, x2off + j] if x2off >= 0 else 1.0)
                block[:, :, k] += a[:, None] * wrow[None, :]
        out[:, out_off : out_off + mul_out * dim3] += block.reshape(Z, -1)
    return out


class SecondPart:
    """The tables of a plan's second part: forward, weight gradient and operand gradients from whole paths."""

    def __init__(self, plan: np.ndarray):
        assert plan[0] == MAGIC and len(plan) == plan[6]
        self.plan = plan
        h = [int(v) for v in plan[int(plan[-1]) : int(plan[-1]) + 14]]
        self.d1max, self.d3max, self.covered, self.swapped = h[8], h[9], h[11], h[12]
        rows = lambda n, at, width: plan[at : at + n * width].reshape(n, width).tolist()      # noqa: E731
        self.groups, self.chunks, self.paths = rows(h[0], h[1], 6), rows(h[2], h[3], 6), rows(h[4], h[5], 16)
        self.in_groups = rows(h[6], h[7], 5)
        assert h[13] == sum(c[2] for c in self.chunks)
        self.in_paths = plan[h[10] : h[10] + sum(g[4] for g in self.in_groups)].tolist()

    def _segment(self, at: int, n: int):
        a, b = int(self.plan[at + n]), int(self.plan[at + n + 1])
        return [(int(self.plan[q]), _i2f(self.plan[q + 1])) for q in range(a, b, 2)]

    def _coupled(self, path, x1, x2, x1off: int, channels: int, x2off: int) -> np.ndarray:
        """A[z, u, k] of `channels` channels: T[z, k, i] = sum_j C_ijk x2[z, j], A = T x1 (Linear: the coefficient times x1)."""
        d1, d3 = path[0], path[2]
        x = x1[:, x1off : x1off + channels * d1].reshape(-1, channels, d1)
        if x2off < 0:
            return _i2f(path[15]) * x
        t = np.zeros((len(x1), d3, d1))
        for k in range(d3):
            for i in range(d1):
                for j, c in self._segment(path[5], k * d1 + i):
                    t[:, k, i] += c * x2[:, x2off + j]
        return np.einsum("zki,zui->zuk", t, x)

    def _walk(self, x1, x2):
        """(group, A of the chunk, flat weight indices [channel, output channel]) of every chunk; T is kept as the kernels do."""
        x1, x2 = (x2, x1) if self.swapped else (x1, x2)
        for out_off, mo, d3, first, n, _ in self.groups:
            t_of = None
            for pid, x1off, channels, x2off, wbase, fresh in self.chunks[first : first + n]:
                path = self.paths[pid]
                assert fresh or t_of == (pid, x2off)
                t_of = (pid, x2off)
                idx = wbase + path[3] * np.arange(channels)[:, None] + path[4] * np.arange(mo)[None, :]
                yield (out_off, mo, d3), self._coupled(path, x1, x2, x1off, channels, x2off), idx

    def forward(self, x1, x2, W) -> np.ndarray:
        out = np.zeros((len(x1), int(self.plan[3])))
        for (off, mo, d3), a, idx in self._walk(x1, x2):
            out[:, off : off + mo * d3] += np.einsum("zuk,uw->zwk", a, W[idx]).reshape(len(x1), -1)
        return out

    def weight_gradient(self, x1, x2, g, numel: int) -> np.ndarray:
        gw = np.zeros(numel)
        for (off, mo, d3), a, idx in self._walk(x1, x2):
            np.add.at(gw, idx, np.einsum("zuk,zwk->uw", a, g[:, off : off + mo * d3].reshape(-1, mo, d3)))
        return gw

    def operand_gradients(self, x1, x2, W, g):
        if self.swapped:
            x1, x2 = x2, x1
        g1, g2 = np.zeros_like(x1), np.zeros_like(x2)
        for x1off, m1, d1, first, n in self.in_groups:
            for pid in self.in_paths[first : first + n]:
                _, d2, d3, su, sw, ki, jj, px1, pm1, x2off, m2, out_off, mo, wbase, sv, _ = path = self.paths[pid]
                assert (px1, pm1, path[0]) == (x1off, m1, d1)
                x, gg = x1[:, x1off : x1off + m1 * d1].reshape(-1, m1, d1), g[:, out_off : out_off + mo * d3].reshape(-1, mo, d3)
                for v in range(m2):
                    w = W[wbase + v * sv + su * np.arange(m1)[:, None] + sw * np.arange(mo)[None, :]]
                    q = np.einsum("uw,zwk->zuk", w, gg)
                    m = np.einsum("zui,zuk->zik", x, q).reshape(len(x1), -1)
                    for j in range(d2):
                        for at, c in self._segment(jj, j):
                            g2[:, x2off + v * d2 + j] += c * m[:, at]
                    for k in range(d3):
                        for i in range(d1):
                            t = sum(c * x2[:, x2off + v * d2 + j] for j, c in self._segment(ki, k * d1 + i))
                            g1[:, x1off : x1off + m1 * d1].reshape(-1, m1, d1)[:, :, i] += np.reshape(t, (-1, 1)) * q[:, :, k]
        return (g2, g1) if self.swapped else (g1, g2)


def _ins(tp):
    return [(i.i_in1, i.i_in2, i.i_out, i.connection_mode, i.has_weight) for i in tp.instructions]


def _oracle_tp(tp, x1, x2, w):
    return orc.tensor_product(str(tp.irreps_in1), str(tp.irreps_in2), str(tp.irreps_out), _ins(tp), x1, x2, w,
                              tp.shared_weights, path_weights=[i.path_weight for i in tp.instructions])


def test_uvw_plan_matches_oracle():
    torch.manual_seed(0)
    tp = o3.FullyConnectedTensorProduct("3x0e+2x1o+4x2e+1x1e", "2x0e+3x1o+1x2e", "5x0e+2x1o+3x2e+2x1e+1x3o")
    x1, x2 = torch.randn(9, tp.irreps_in1.dim, dtype=torch.float64), torch.randn(9, tp.irreps_in2.dim, dtype=torch.float64)
    w = tp.weight.detach().double()
    got = run_plan(tp._plan_host, x1.numpy(), x2.numpy(), w.numpy())
    # the plan stores its coefficients in fp32
    assert rel_err(torch.from_numpy(got), _oracle_tp(tp, x1, x2, w)) < 1e-6


@pytest.mark.parametrize("layout,swapped", [
    (("3x0e+2x1o+4x2e+1x1e", "2x0e+3x1o+1x2e", "5x0e+2x1o+3x2e+2x1e+1x3o"), False),
    (("33x0e+65x1o", "1x0e+2x1o", "40x0e+1x1o+2x1e"), False),                   # more than a chunk of channels
    (("1x0e+2x1o", "33x0e+65x1o", "40x0e+1x1o+2x1e"), True),                    # the second operand's channels taken by 32
    (("4x0e+4x1o", "4x0e+4x1o", "2x0e+3x1e"), False),                           # as many either way
    (("1x0e+2x2e", "20x0e+20x4e", "5x0e+6x2e"), False),                         # l = 4 stays second
    (("1x0e+2x4e", "20x0e+20x4e", "5x0e+6x2e"), True),                          # l = 4 either way
    (("2x4e+1x0e+3x5o", "1x4e+2x0e", "2x4e+1x0e+0x1o"), False)])                # an operand block no path leaves
def test_second_part_of_product_plans(layout, swapped):
    """What the register-tile kernels read: forward and all gradients against autograd through the oracle."""
    torch.manual_seed(0)
    tp = o3.FullyConnectedTensorProduct(*layout)
    x1, x2 = (torch.randn(5, d, dtype=torch.float64, requires_grad=True) for d in (tp.irreps_in1.dim, tp.irreps_in2.dim))
    w = tp.weight.detach().double().requires_grad_(True)
    ref = _oracle_tp(tp, x1, x2, w)
    go = torch.randn_like(ref)
    want = [ref.detach()] + list(torch.autograd.grad(ref, [w, x1, x2], go))
    part = SecondPart(tp._plan_host)
    a, b, ww, g = (t.detach().numpy() for t in (x1, x2, w, go))
    got = [part.forward(a, b, ww), part.weight_gradient(a, b, g, len(ww)), *part.operand_gradients(a, b, ww, g)]
    for x, y in zip(got, want):
        assert rel_err(torch.from_numpy(x), y) < 1e-6        # (the coefficients are fp32)
    assert bool(part.swapped) == swapped
    first, where = (tp.irreps_in2, "i_in2") if swapped else (tp.irreps_in1, "i_in1")
    live = {getattr(i, where) for i in tp.instructions if 0 not in i.path_shape}
    assert bool(part.covered) == all(n in live for n, m in enumerate(first) if m.dim > 0)


def test_second_part_of_linear_plans():
    torch.manual_seed(1)
    lin = o3.Linear("6x0e+4x1o+3x2e+35x0e", "5x0e+2x0e+4x1o+3x1o+3x0o")
    x = torch.randn(7, lin.irreps_in.dim, dtype=torch.float64, requires_grad=True)
    w = lin.weight.detach().double().requires_grad_(True)
    ref = orc.linear(str(lin.irreps_in), str(lin.irreps_out), x, w)
    go = torch.randn_like(ref)
    gx, gw = torch.autograd.grad(ref, [x, w], go)
    forward, back = SecondPart(lin._plan_host), SecondPart(lin._plan_t_host)
    a, ww, g = (t.detach().numpy() for t in (x, w, go))
    assert rel_err(torch.from_numpy(forward.forward(a, None, ww)), ref.detach()) < 1e-6
    assert rel_err(torch.from_numpy(forward.weight_gradient(a, None, g, len(ww))), gw) < 1e-6
    assert rel_err(torch.from_numpy(back.forward(g, None, ww)), gx) < 1e-6
    assert not lin._reads_all


def test_linear_plans_forward_and_transposed_with_mixed_multiplicities():
    torch.manual_seed(1)
    lin = o3.Linear("6x0e+4x1o+3x2e", "5x0e+2x0e+4x1o+3x2e+1x1o")   # two outputs of different width from one input
    x = torch.randn(7, lin.irreps_in.dim, dtype=torch.float64, requires_grad=True)
    w = lin.weight.detach().double()
    ref = orc.linear(str(lin.irreps_in), str(lin.irreps_out), x, w)
    got = run_plan(lin._plan_host, x.detach().numpy(), None, w.numpy())
    assert rel_err(torch.from_numpy(got), ref.detach()) < 1e-6
    go = torch.randn_like(ref)
    ref.backward(go)
    # the transposed plan may hold several groups per input irrep (one per output multiplicity): accumulated
    gx = run_plan(lin._plan_t_host, go.numpy(), None, w.numpy())
    assert rel_err(torch.from_numpy(gx), x.grad) < 1e-6
    strides = {int(lin._plan_t_host[int(lin._plan_t_host[7]) + 6 * g + 5]) for g in range(int(lin._plan_t_host[4]))}
    assert {5, 2} <= strides


def test_operand_gradients_are_transposed_products():
    """`TensorProduct._vjp_module` / `_vjp_weights` against autograd through the oracle (fp64, exact up to rounding)."""
    torch.manual_seed(2)
    tp = o3.FullyConnectedTensorProduct("5x0e+3x1o+2x2e+1x3o", "2x0e+3x1o+1x2e", "4x0e+2x0o+3x1o+2x1e+1x2e")
    Z = 6
    x = torch.randn(Z, tp.irreps_in1.dim, dtype=torch.float64, requires_grad=True)
    y = torch.randn(Z, tp.irreps_in2.dim, dtype=torch.float64, requires_grad=True)
    w = tp.weight.detach().double()
    go = torch.randn(Z, tp.irreps_out.dim, dtype=torch.float64)
    _oracle_tp(tp, x, y, w).backward(go)
    m0, m1 = tp._vjp_module(0), tp._vjp_module(1)
    assert set(m0._vjp_signs) <= {1.0, -1.0} and -1.0 in m0._vjp_signs     # odd permutations of (1, 1, 1)-like triples
    g1 = _oracle_tp(m0, go, y.detach(), tp._vjp_weights(0, w))
    g2 = _oracle_tp(m1, x.detach(), go, tp._vjp_weights(1, w))
    assert rel_err(g1, x.grad) < 1e-12
    assert rel_err(g2, y.grad) < 1e-12
    # and through the plans the kernels would read
    g1p = run_plan(m0._plan_host, go.numpy(), y.detach().numpy(), tp._vjp_weights(0, w).numpy())
    assert rel_err(torch.from_numpy(g1p), x.grad) < 1e-6


def test_linear_plan_rejects_nothing_it_accepts_in_forward():
    # empty instruction lists and zero-multiplicity irreps build (degenerate) plans
    plan, written = linear_plan(o3.Irreps("0x0e+2x1o"), o3.Irreps("3x1o"), o3.Linear("0x0e+2x1o", "3x1o").instructions)
    assert written == [0] and int(plan[4]) == 1


def _first_part(plan: np.ndarray) -> np.ndarray:
    """The plan as it was before there was a second part."""
    old = plan[: int(plan[10]) + _cg_words(plan)].copy()
    old[0], old[6] = 0x65336250, len(old)
    return old


def _cg_words(plan: np.ndarray) -> int:
    paths = [int(plan[int(plan[9]) + p]) for p in range(int(plan[5]))] + [int(plan[10])]
    return max([3 * int(plan[a] + plan[a + 1]) for p, q in zip(paths, paths[1:]) for a in range(p, q, 2)], default=0)


def test_plans_without_a_second_part():
    """Modules saved with such plans get new ones when they are loaded; the entry point that needs the second part refuses."""
    import pickle

    from e3nn_b200 import _lib

    tp, lin = o3.FullyConnectedTensorProduct("3x0e+2x1o", "1x0e+1x1o", "2x0e+3x1o"), o3.Linear("3x0e+2x1o", "4x0e+2x1o")
    written, plans = tp._uvw_written, (tp._plan_host, lin._plan_host, lin._plan_t_host)
    tp._plan_host, lin._plan_host, lin._plan_t_host = (_first_part(p) for p in plans)
    del lin._reads_all
    x1, x2 = np.random.randn(4, tp.irreps_in1.dim), np.random.randn(4, tp.irreps_in2.dim)
    w = tp.weight.detach().double().numpy()
    assert np.array_equal(run_plan(tp._plan_host, x1, x2, w), run_plan(plans[0], x1, x2, w))
    tp2, lin2 = (pickle.loads(pickle.dumps(m)) for m in (tp, lin))
    for got, want in zip((tp2._plan_host, lin2._plan_host, lin2._plan_t_host), plans):
        assert np.array_equal(got, want)
    assert lin2._reads_all and tp2._uvw_written == written
    core, host = _lib.core(), tp._plan_host.ctypes.data
    assert core.e3b_dense_bwd_x_supported(host) == 0 and core.e3b_dense_bwd_x_supported(plans[0].ctypes.data) == 1
    assert core.e3b_dense_bwd_x(host, None, None, None, None, None, None, None, 5, None) == -1


# ----------------------------------------------------------------------------- planner of the post-coupling 'uvw' kernel
UVW_POST_LAYOUTS = [
    ("128x0e+64x1o+32x2e", "0e+1o+2e+3o", "128x0e+64x1o+32x2e"),
    ("32x0e+32x1o+32x2e", "1x0e+1x1o+1x2e", "32x0e+32x1o+32x2e"),
    ("64x0e+64x1o+64x2e", "0e+1o+2e", "48x0e+32x1o+16x2e"),
    ("96x0e+32x1e+32x2e+32x3o", "0e+1o+2e+3o", "64x0e+32x1o+32x2e+16x3o"),
    ("32x0e+32x1o", "0e+1o", "256x0e+16x1o"),
    ("64x0e+64x1o+64x2e+64x3o", "0e", "64x0e+64x1o+64x2e+64x3o"),
]


def test_uvw_post_plan_covers_every_path_and_fits_the_sm():
    from e3nn_b200 import o3
    from e3nn_b200.codegen import uvw_post

    for layout in UVW_POST_LAYOUTS:
        tp = o3.FullyConnectedTensorProduct(*layout, math_mode="tf32")
        groups = uvw_post.plan_groups(tp._spec)
        assert groups is not None, layout
        covered = {}
        for g in groups:
            assert g.smem_bytes() <= uvw_post.SMEM_LIMIT and g.nacc() <= uvw_post.MAX_ACC_REGS
            assert g.nstage() >= max(b.d1 for b in g.blocks) + 1          # a chunk's component tiles fit the ring together
            assert g.nslots * g.slot_cols <= uvw_post.TMEM_COLS
            for b in g.blocks:
                assert b.ncols <= uvw_post.MAX_N and b.ncols % 16 == 0
                col = 0
                for p in b.paths:                                          # the paths of a block lie side by side
                    m = g.members[p.member]
                    assert p.coloff == col
                    col += m.width
                    covered.setdefault(p.index, []).append((m.col0, m.width))
                assert col == b.ncols
            for j in g.jobs:
                assert 0 <= j.slot0 and j.slot0 + j.nslot <= g.nslots
                assert j.cols(g.blocks) <= j.nslot * g.slot_cols
            # every stage the producers emit is consumed by exactly one job, in the producers' order
            assert sum(len(j.comps) * j.nchunk for j in g.jobs) == g.tiles_per_row_tile()
        # every live path: all of its output channels, once
        for n, ins in tp._spec.live_instructions():
            mul_o = tp._spec.irreps_out[ins.i_out].mul
            slabs = sorted(covered[n])
            assert slabs[0][0] == 0 and sum(w for _, w in slabs) == mul_o
            assert all(a[0] + a[1] == b[0] for a, b in zip(slabs, slabs[1:]))


def test_uvw_post_slot_schedule_is_safe():
    """The issuing thread may overwrite a tensor-memory slot only after the epilogue has read the job that held it,
    and it learns that from mbarrier phases (one bit): replay the static schedule over several row tiles and check
    that (a) every job's slots are free of unread accumulators once its waits are done, and (b) the completions of
    every barrier are observed one by one, in order, before the next job that arrives on that barrier is issued."""
    from e3nn_b200 import o3
    from e3nn_b200.codegen import uvw_post

    for layout in UVW_POST_LAYOUTS:
        tp = o3.FullyConnectedTensorProduct(*layout, math_mode="tf32")
        for g in uvw_post.plan_groups(tp._spec):
            holder = [None] * g.nslots              # (tile, job) whose accumulators a slot holds, None once observed as read
            observed = [0] * g.nslots               # completions of empty[b] the issuing thread has seen
            produced = [0] * g.nslots               # jobs issued so far whose first slot is b (= arrivals the barrier will get)
            for tile in range(4):
                for ji, j in enumerate(g.jobs):
                    for bar, idx, prev in j.waits:
                        if prev and tile == 0:
                            continue                # nothing ran before the first tile
                        t = tile - 1 if prev else tile
                        n = t * g.uses[bar] + idx   # the completion this wait is for
                        assert n == observed[bar], (layout, tile, ji, bar)       # in order, none skipped: parity is enough
                        assert n < produced[bar]                                    # that job has been issued
                        observed[bar] += 1
                        for s in range(g.nslots):   # its slots are free now
                            if holder[s] is not None and holder[s][2] == (bar, n):
                                holder[s] = None
                    for s in range(j.slot0, j.slot0 + j.nslot):
                        assert holder[s] is None, (layout, tile, ji, s, holder[s])
                    n_mine = tile * g.uses[j.slot0] + j.use_idx
                    assert n_mine == produced[j.slot0]                             # the epilogue's phase arithmetic
                    assert observed[j.slot0] == produced[j.slot0]                  # no unobserved completion on my barrier
                    produced[j.slot0] += 1
                    for s in range(j.slot0, j.slot0 + j.nslot):
                        holder[s] = (tile, ji, (j.slot0, n_mine))


def test_transposed_linear_swaps_operands_only_where_it_pays():
    """Groups of a transposed Linear run with swapped MMA operands when 2l+1 is 3 or 5 and the group is a whole number
    of 128-channel MMA tiles; forward Linears, scalars and 2l+1 = 7 keep the row order."""
    from e3nn_b200 import o3

    lin = o3.Linear("128x0e+128x1o+256x2e+128x3o", "64x0e+64x1o+32x2e+32x3o", math_mode="tf32x3")
    assert [(g.n, g.dim, g.swap) for g in lin._tc_bwd.groups] == [(128, 1, False), (128, 3, True), (256, 5, True), (128, 7, False)]
    assert not any(g.swap for g in lin._tc_fwd.groups)
    small = o3.Linear("64x0e+64x1o", "64x0e+64x1o", math_mode="tf32x3")
    assert not any(g.swap for g in small._tc_bwd.groups)          # 64 channels: half an MMA tile
    for g in lin._tc_bwd.groups:
        assert not (g.swap and g.staged_epilogue())


def test_spherical_harmonics_module_is_kept_by_its_arguments():
    """The functional form keeps one module per set of arguments: equal arguments share it, different types do not."""
    from e3nn_b200 import o3
    from e3nn_b200.o3._spherical_harmonics import _module

    irreps = o3.Irreps("1x0e+1x1o+1x2e")
    kept = _module(irreps, o3.Irreps, True, "component")
    assert kept is _module(o3.Irreps("0e+1o+2e"), o3.Irreps, True, "component")
    assert kept is not _module(irreps, o3.Irreps, False, "component") and kept is not _module(irreps, o3.Irreps, True, "norm")
    as_list = _module((0, 1, 2), list, True, "component")
    assert as_list is not kept and as_list._ls_list == [0, 1, 2] and _module((2, 0), list, True, "component")._ls_list == [2, 0]
    assert _module(2, int, True, "component")._ls_list == [2] and _module("2e", str, True, "component").irreps_out == o3.Irreps("1x2e")
