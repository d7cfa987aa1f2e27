"""PCG with the matrix resident in shared memory (k_pcg_persist, node-row
systems of up to about 3 million values) against the plain-CSR PCG of the same
library, which runs a kernel per part of an iteration: one CTA and many,
constrained and shuffled nodes, several launches per solve, and the sizes at
which a share just fits or does not.

Both stop at a squared relative residual of 1e-20 in the D^-1 norm; their
iterates then differ by at most sqrt(cond) * 1e-10 relative in the energy norm:
1e-7 of the largest entry at these condition numbers (below 1e5)."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr())


def system(kind, dims, fixed="clamp", shuffle=False, seed=0):
    from fea_b200 import DevicePlan
    from fea_b200.meshes import hex_block, tet_block
    rng = np.random.default_rng(seed)
    X, el = (hex_block if kind == "C3D8" else tet_block)(0, dims=dims)
    X = X + rng.uniform(-0.05, 0.05, X.shape) / max(dims)
    N = len(X)
    mask = np.full(N, 7, np.uint8)
    first = np.nonzero(X[:, 0] < 0.5 / dims[0])[0]
    mask[first] = 0 if fixed == "clamp" else 2         # roller: y free on the plane
    if fixed == "roller":
        mask[first[0]] = 0
    if shuffle:
        perm = rng.permutation(N)
        inv = np.empty(N, np.int64)
        inv[perm] = np.arange(N)
        X, el, mask = X[perm], inv[el], mask[perm]
    P = DevicePlan(X, mask, [(kind, el)])
    K = torch.empty(P.nnz, dtype=torch.float64, device="cuda")
    P.assemble_volume(0, 1.0, 10.0, P.zeros(P.ndof), K=K, R=P.zeros(P.ndof))
    b = torch.from_numpy(rng.normal(size=P.ndof)).cuda()
    return P, K, b


def relres(P, K, x, b):
    r = b - P.spmv(K, x)
    diag = torch.zeros_like(b)
    ip, ix = P.indptr, P.indices.long()
    rows = torch.repeat_interleave(torch.arange(P.ndof, device="cuda"), ip[1:] - ip[:-1])
    diag[rows[rows == ix]] = K[rows == ix]
    return float((r * r / diag).sum() / (b * b / diag).sum())


CASES = [("C3D8", (1, 1, 1), "clamp", False), ("C3D4", (1, 1, 1), "roller", False), ("C3D8", (2, 3, 2), "roller", True),
         ("C3D4", (5, 4, 3), "clamp", True), ("C3D8", (9, 8, 7), "roller", False), ("C3D4", (24, 6, 5), "clamp", False),
         ("C3D8", (23, 22, 22), "clamp", False), ("C3D8", (26, 26, 26), "clamp", False), ("C3D4", (30, 30, 30), "roller", True)]


@pytest.mark.parametrize("kind,dims,fixed,shuffle", CASES)
def test_matches_plain_csr_pcg(kind, dims, fixed, shuffle):
    P, K, b = system(kind, dims, fixed, shuffle)
    xa, xb, xc = (torch.zeros_like(b) for _ in range(3))
    ia, ra, sa = P.pcg(K, b, xa, 1e-20, 20000, check_every=7)
    ib, rb, sb = P.pcg(K, b, xb, 1e-20, 20000, check_every=7, generic=True)
    assert sa == sb == 0 and ra < 1e-20
    assert abs(ia - ib) <= 2 + ib // 50
    assert relres(P, K, xa, b) < 1e-18                 # (recurrence and true residual differ by round-off)
    assert float((xa - xb).abs().max()) <= 1e-7 * float(xb.abs().max())
    P.pcg(K, b, xc, 1e-20, 20000, check_every=50)
    assert torch.equal(xa, xc)                         # bitwise the same from run to run


@pytest.mark.parametrize("kind,dims,resident", [("C3D8", (1, 1, 1), True), ("C3D4", (24, 6, 5), True),
                                                ("C3D8", (23, 22, 22), True), ("C3D8", (26, 26, 26), False)])
def test_which_systems_are_resident(kind, dims, resident):
    """A resident solve of 300 iterations is a few launches, the kernels per
    part are two an iteration."""
    from fea_b200 import _lib as L
    P, K, b = system(kind, dims)
    n0 = L.fea_launch_count()
    assert P.pcg(K, b, torch.zeros_like(b), 1e-300, 300)[0] <= 300
    n = L.fea_launch_count() - n0
    assert n <= 20 if resident else n >= 600


def test_caps_guesses_and_breakdown():
    from fea_b200 import _lib as L
    P, K, b = system("C3D8", (10, 9, 9))
    x = torch.zeros_like(b)
    assert P.pcg(K, b, x, 1e-30, 0)[0] == 0 and not x.any()
    for cap in (1, 3, 600):                            # 600: more than one launch
        x = torch.zeros_like(b)
        it, rr, st = P.pcg(K, b, x, 1e-300, cap)
        assert (it, st) == (cap, L.FEA_ENOTCONV)
    it, rr, st = P.pcg(K, b, x, 1e-16, 1000)           # from the converged iterate
    assert st == 0 and it <= 1
    z = torch.zeros_like(b)
    assert P.pcg(K, z, z.clone(), 1e-20, 100)[0] == 0
    x1, x2 = torch.randn_like(b), torch.zeros_like(b)  # a start that is not zero
    P.pcg(K, b, x1, 1e-22, 5000)
    P.pcg(K, b, x2, 1e-22, 5000)
    assert float((x1 - x2).abs().max()) <= 1e-7 * float(x2.abs().max())
    it, rr, st = P.pcg(-K, b, torch.zeros_like(b), 1e-20, 100, raise_on_breakdown=False)
    assert st == L.FEA_EBREAKDOWN and it == 0
    bad = b.clone()
    bad[5] = float("nan")
    assert P.pcg(K, bad, torch.zeros_like(b), 1e-20, 100, raise_on_breakdown=False)[2] == L.FEA_EBREAKDOWN


@pytest.mark.parametrize("kind,dims,extra", [("C3D8", (1, 1, 1), 1), ("C3D4", (5, 4, 3), 40), ("C3D8", (12, 9, 8), 300)])
def test_free_nodes_without_elements(kind, dims, extra):
    """Free nodes that no element holds (empty rows, a zero right-hand side) at
    the start, in the middle and at the end of the numbering, alone and in
    runs: they stay at their start value 0 and the others' solution is that
    of the mesh without them."""
    from fea_b200 import DevicePlan
    from fea_b200.meshes import hex_block, tet_block
    P, K, b = system(kind, dims, "roller")
    _, el = (hex_block if kind == "C3D8" else tet_block)(0, dims=dims)
    X, mask = P.X.cpu().numpy(), P.mask.cpu().numpy()
    N = len(X)
    at = np.unique(np.concatenate([[0, N // 2, N], np.linspace(1, N - 1, 5).astype(int)]))    # runs before these nodes
    new = np.zeros(N, np.int64)
    shift = 0
    keep = np.ones(N + extra * len(at), bool)
    for n in range(N + 1):
        if n in at:
            keep[n + shift:n + shift + extra] = False
            shift += extra
        if n < N:
            new[n] = n + shift
    X2 = np.zeros((len(keep), 3))
    m2 = np.where(np.arange(len(keep)) % 3 == 0, 2, 7).astype(np.uint8)     # (some of them free in y only)
    X2[keep], m2[keep] = X, mask
    Q = DevicePlan(X2, m2, [(kind, new[el])])
    assert Q.nnz == P.nnz
    f = ((m2[:, None] >> np.arange(3)) & 1).astype(bool)
    rows = torch.from_numpy(np.nonzero(np.repeat(keep[:, None], 3, 1)[f])[0]).cuda()
    b2 = Q.zeros(Q.ndof)
    b2[rows] = b
    x, xa, xb = torch.zeros_like(b), torch.zeros_like(b2), torch.zeros_like(b2)
    it = P.pcg(K, b, x, 1e-20, 20000)
    ia = Q.pcg(K, b2, xa, 1e-20, 20000)
    ib = Q.pcg(K, b2, xb, 1e-20, 20000, generic=True)
    assert it[2] == ia[2] == ib[2] == 0 and abs(ia[0] - ib[0]) <= 2 + ib[0] // 50
    other = torch.ones_like(b2, dtype=torch.bool)
    other[rows] = False
    assert not xa[other].any() and not xb[other].any()
    for y in (xa[rows], xb[rows]):
        assert float((y - x).abs().max()) <= 1e-7 * float(x.abs().max())


@pytest.mark.parametrize("shift", [0, 1])
def test_work_buffer_bounds_and_alignment(shift):
    """The buffer's tail is untouched, also where the work pointer is not
    16-byte aligned."""
    from fea_b200 import _lib as L
    P, K, b = system("C3D4", (7, 6, 5), "roller", True)
    wl = int(L.fea_pcg_work_len(P.ndof))
    buf = torch.full((wl + 64 + shift,), 3.5, dtype=torch.float64, device="cuda")
    xb = torch.full((P.ndof + 32,), 0.0, dtype=torch.float64, device="cuda")
    it, rr = C.c_int32(0), C.c_double(0)
    st = L.fea_pcg_solve_nodes(C.byref(P.nodes), ptr(P.indices), ptr(K), ptr(b), ptr(xb), 1e-20, 5000, 20,
                               C.c_void_p(buf.data_ptr() + 8 * shift), wl, C.byref(it), C.byref(rr),
                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0 and bool((buf[wl + shift:] == 3.5).all()) and not xb[P.ndof:].any()
    if shift:
        assert float(buf[0]) == 3.5
    x = torch.zeros_like(b)
    P.pcg(K, b, x, 1e-20, 5000, generic=True)
    assert float((xb[:P.ndof] - x).abs().max()) <= 1e-7 * float(x.abs().max())


def test_solves_on_two_streams():
    P, K, b = system("C3D4", (20, 6, 5))
    Q, K2, b2 = system("C3D8", (12, 9, 8))
    ref = [torch.zeros_like(b), torch.zeros_like(b2)]
    P.pcg(K, b, ref[0], 1e-20, 5000)
    Q.pcg(K2, b2, ref[1], 1e-20, 5000)
    import threading
    out = [torch.zeros_like(b), torch.zeros_like(b2)]
    torch.cuda.synchronize()

    def go(k, p, kk, bb):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                out[k].zero_()
                p.pcg(kk, bb, out[k], 1e-20, 5000)
    th = [threading.Thread(target=go, args=a) for a in ((0, P, K, b), (1, Q, K2, b2))]
    [t.start() for t in th]
    [t.join() for t in th]
    assert torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])


def test_systems_of_different_size_on_two_threads():
    """One thread solves a system of nearly 3 million values, whose iterations
    take several launches of most of an SM's shared memory, while another
    solves one of a few rows over and over: both as alone, bit for bit."""
    import threading
    from fea_b200 import _lib as L
    P, K, b = system("C3D8", (23, 22, 22))
    Q, K2, b2 = system("C3D8", (1, 1, 1), "roller")
    assert 2_500_000 < P.nnz < 3_000_000 and Q.ndof < 24
    ref = [torch.zeros_like(b), torch.zeros_like(b2)]
    assert P.pcg(K, b, ref[0], 1e-300, 1000)[::2] == (1000, L.FEA_ENOTCONV)   # (about 190 iterations per launch)
    assert Q.pcg(K2, b2, ref[1], 1e-20, 500)[2] == 0
    torch.cuda.synchronize()
    stop, count, errors = threading.Event(), [0], []

    def small():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                while not stop.is_set():
                    x = torch.zeros_like(b2)
                    Q.pcg(K2, b2, x, 1e-20, 500)
                    assert torch.equal(x, ref[1])
                    count[0] += 1
        except BaseException as e:
            errors.append(e)
    th = threading.Thread(target=small)
    th.start()
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(6):
                x = torch.zeros_like(b)
                assert P.pcg(K, b, x, 1e-300, 1000)[::2] == (1000, L.FEA_ENOTCONV)
                assert torch.equal(x, ref[0])
    finally:
        stop.set()
        th.join()
    assert not errors and count[0] > 0
