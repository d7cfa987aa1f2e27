"""The FP32 inner solver on the padded node layout (fea_f32_layout_fill,
fea_pcg_solve_mixed_nodes32): the layout holds the plan's FP32 values and
columns (padding zeros), the mixed solve meets its FP64 stop test and the
direct solution to 1e-8 with and without inner_tol, and the Newton solver's mixed mode uses
it."""
import numpy as np
import pytest
import torch

from oracle import fea_oracle as O
from tests.helpers import fea_model, rel

pytestmark = pytest.mark.gpu


def test_padded_layout_holds_the_plan_matrix(golden):
    g = golden("hex5")
    c, e, _ = fea_model(g, "C3D8")
    c.initialize()
    P = c.assembly.plan
    R, K = c.assembly.assemble_csr(torch.from_numpy(g["state"]).cuda())
    desc, cbase, qbase, cols, vals = P.f32_layout()
    P.fill_f32(K)
    ip, ix = P.indptr.cpu().numpy(), P.indices.cpu().numpy()
    Kc = K.cpu().numpy()
    mask, rowlen, rdof = P.mask.cpu().numpy(), P.rowlen.cpu().numpy(), P.rdof.cpu().numpy()
    cb, qb, cl, vl = cbase.cpu().numpy(), qbase.cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy()
    assert np.all(cb % 4 == 0) and np.all(qb % 4 == 0)
    for nd in range(P.n_nodes):
        if mask[nd] == 0:
            assert cb[nd + 1] == cb[nd]
            continue
        L, L4 = int(rowlen[nd]), int(cb[nd + 1] - cb[nd])
        assert L4 == (L + 3) // 4 * 4
        f = bin(int(mask[nd])).count("1")
        for j in range(f):
            row = int(rdof[nd]) + j
            a, b = int(ip[row]), int(ip[row + 1])
            assert np.array_equal(cl[cb[nd]:cb[nd] + L], ix[a:b]) and not cl[cb[nd] + L:cb[nd + 1]].any()
            v = vl[qb[nd] + j * L4:qb[nd] + (j + 1) * L4]
            assert np.array_equal(v[:L], Kc[a:b].astype(np.float32)) and not v[L:].any()


@pytest.mark.parametrize("inner_tol", [0.0, 1e-4])
def test_mixed_padded_layout_solve_matches_direct(golden, inner_tol):
    g = golden("hex5")
    c, e, _ = fea_model(g, "C3D8")
    c.initialize()
    P = c.assembly.plan
    R, K = c.assembly.assemble_csr(torch.from_numpy(g["state"]).cuda())
    b = (-R).contiguous()
    x = torch.zeros_like(b)
    it, outer, rr, st = P.pcg_mixed(K, None, b, x, 1e-22, inner_tol, 20000, check_every=20)
    assert st == 0 and outer >= 1
    ip, ix, Kc = P.indptr.cpu(), P.indices.cpu().long(), K.cpu()
    xd = O.direct_solve(ip, ix, Kc, b.cpu())
    # the true FP64 residual meets the stop test (r.D^-1 r)/(b.D^-1 b) < tol,
    # and the displacements are within the 1e-8 of the solver contract
    A = torch.sparse_csr_tensor(ip, ix, Kc, (b.numel(), b.numel()))
    rows = torch.repeat_interleave(torch.arange(b.numel()), ip[1:] - ip[:-1])
    dinv = 1.0 / Kc[ix == rows]
    r = b.cpu() - A @ x.cpu()
    assert float((r * dinv * r).sum() / (b.cpu() * dinv * b.cpu()).sum()) < 1e-20
    assert rel(x, xd) < 1e-8
    if inner_tol > 0:
        x0 = torch.zeros_like(b)
        it0, outer0, _, st0 = P.pcg_mixed(K, None, b, x0, 1e-22, 0.0, 20000, check_every=20)
        assert st0 == 0 and outer <= outer0


def test_newton_mixed_mode_on_padded_layout(golden):
    import fea_b200 as F
    g = golden("hex5")
    c, e, _ = fea_model(g, "C3D8", solver=F.solver.StaticImplicitSolver(rtol=1e-11, maximum_iteration=60,
                                                                          precision="mixed"))
    c.initialize()
    gc = c.solver.solve()
    assert not isinstance(gc, bool)
    assert rel(gc, g["gc_converged"]) < 1e-8


@pytest.mark.parametrize("copies", [2, 60])
def test_search_direction_has_the_same_bits_at_every_size(copies):
    """p = z + beta p is formed in FP64 and rounded once, in the SpMV's gather
    (small systems) as in a kernel of its own (large ones): several copies of
    one system side by side take the steps of the single one (every sum is the
    copies' multiple up to its FP64 rounding), so that the FP32 iterates hold
    the same bits but where 1e-16 in a scalar crosses a rounding boundary, 1e-8
    of them per step."""
    import ctypes as C
    from fea_b200 import _lib as L
    rng = np.random.default_rng(7)
    n1 = 20000
    d, b1 = 2.0 + rng.uniform(0.01, 1.0, n1), rng.normal(size=n1)

    def solve(k):
        n = k * n1
        row = np.arange(n1)
        cols = row[:, None] + np.array([-1, 0, 1])
        ok = (cols >= 0) & (cols < n1)
        vals = np.where(cols == row[:, None], d[:, None], -1.0)
        ip = np.concatenate([[0], np.cumsum(np.tile(ok.sum(1), k))]).astype(np.int64)
        ix = (cols[ok][None, :] + n1 * np.arange(k)[:, None]).reshape(-1).astype(np.int32)
        v = torch.from_numpy(np.tile(vals[ok], k)).cuda()
        ip, ix, b = torch.from_numpy(ip).cuda(), torch.from_numpy(ix).cuda(), torch.from_numpy(np.tile(b1, k)).cuda()
        v32, x = v.float(), torch.zeros(n, dtype=torch.float64, device="cuda")
        w = torch.empty(int(L.fea_pcg_mixed_work_len(n)), dtype=torch.float64, device="cuda")
        it, out, rr = C.c_int32(0), C.c_int32(0), C.c_double(0)
        st = L.fea_pcg_solve_mixed(n, ip.data_ptr(), ix.data_ptr(), v.data_ptr(), v32.data_ptr(), b.data_ptr(), x.data_ptr(),
                                   1e-30, 0.0, 12, 12, w.data_ptr(), w.numel(), C.byref(it), C.byref(out), C.byref(rr),
                                   torch.cuda.current_stream().cuda_stream)
        assert st == L.FEA_ENOTCONV and it.value == 12
        return x.view(k, n1)
    one, many = solve(1), solve(copies)
    assert float((one != 0).double().mean()) > 0.99
    assert float((many != one).double().mean()) < 1e-5


@pytest.mark.parametrize("dims,rows", [((26, 26, 26), 56862), ((27, 27, 27), 63504)])
def test_plan_layout_solve_on_both_sides_of_the_pairs_line(dims, rows):
    """FP32 values in the plan's layout below and above the 60,000 rows from
    which p has an array of its own, against the FP64 solve: both meet the FP64
    stop test at 1e-16 (squared), and the iterates differ by sqrt(cond) of its
    root, below 1e-5 of the largest entry."""
    from fea_b200 import DevicePlan
    from fea_b200.meshes import hex_block
    X, el = hex_block(0, dims=dims)
    mask = np.full(len(X), 7, np.uint8)
    mask[X[:, 0] == 0] = 0
    P = DevicePlan(X, mask, [("C3D8", el)])
    assert P.ndof == rows
    K = P.zeros(P.nnz)
    P.assemble_volume(0, 1.0, 10.0, P.zeros(P.ndof), K=K)
    b = torch.from_numpy(np.random.default_rng(1).normal(size=P.ndof)).cuda()
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    it, out, rr, st = P.pcg_mixed(K, P.to_f32(K), b, x, 1e-16, 0.0, 20000, check_every=50)
    assert st == 0 and out >= 1 and rr < 1e-16
    assert P.pcg(K, b, y, 1e-22, 20000)[2] == 0
    assert float((x - y).abs().max()) <= 1e-5 * float(y.abs().max())
