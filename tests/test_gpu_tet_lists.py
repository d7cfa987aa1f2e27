"""C3D4 tangent and residual by column lists (k_tet_rk) against the rank-round
kernel, which the same entry point takes for a descriptor without lists:
chunks with one and with many nodes, a node shared by 120 tetrahedra, partly
fixed nodes, a doubled element, accumulate, no residual, and the
element residual.  Each entry sums the same contributions in the same order;
the strips differ by the rounding of g_a . g_b (formed as f_a . q_b): 1e-12 of the
largest entry bounds it."""
import ctypes as C

import numpy as np
import pytest
import torch

gpu = pytest.mark.gpu

TOL = 1e-12


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def fan(n):
    """n tetrahedra around the axis (0, 1): both axis nodes lie in all of them."""
    t = 2 * np.pi * np.arange(n) / n
    X = np.concatenate([[[0, 0, -1.0], [0, 0, 1.0]], np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(3 * t)], 1)])
    r = 2 + np.arange(n)
    el = np.stack([np.zeros(n, int), r, 2 + (np.arange(n) + 1) % n, np.ones(n, int)], 1)
    return X, el


def mesh(kind):
    from fea_b200.meshes import tet_block
    rng = np.random.default_rng(1)
    if kind == "fan":
        X, el = fan(120)
    else:
        X, el = tet_block(0, dims=kind)
        X = X + rng.uniform(-0.05, 0.05, X.shape) / max(kind)
        perm = rng.permutation(len(X))
        inv = np.empty(len(X), np.int64)
        inv[perm] = np.arange(len(X))
        X, el = X[perm], inv[el]
    return X, el


@gpu
@pytest.mark.parametrize("kind", [(1, 1, 1), (2, 1, 1), (5, 4, 3), (9, 8, 7), "fan"])
@pytest.mark.parametrize("repeat", [False, True])
def test_lists_match_rank_rounds(kind, repeat):
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    X, el = mesh(kind)
    N = len(X)
    if repeat:
        el = np.concatenate([el, el[-1:]])        # a doubled element
    mask = np.full(N, 7, np.uint8)
    mask[N // 2], mask[N // 3], mask[-1] = 0, 5, 2
    P = DevicePlan(X, mask, [("C3D4", el)])
    g = P.groups[0]
    gc = torch.from_numpy(np.random.default_rng(2).normal(0, 5e-3 / (1 if kind == "fan" else max(kind)), P.ndof)).cuda()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert P.tangent_lists(0)[0].clist_dev
    old = L.Group()
    C.memmove(C.byref(old), C.byref(g.desc), C.sizeof(L.Group))
    old.clist_dev = None
    for acc in (0, 1):
        for with_R in (True, False):
            for with_e in (False, True):
                out = []
                for d in (old, g.desc):
                    pad = torch.full((P.nnz + 64,), 0.5, dtype=torch.float64, device="cuda")
                    R = torch.full((P.ndof + 64,), 0.25, dtype=torch.float64, device="cuda")
                    eR = torch.zeros(12 * g.ne, dtype=torch.float64, device="cuda")
                    L.check(L.fea_assemble_volume(C.byref(P.nodes), C.byref(d), 1.0, 30.0, ptr(gc), ptr(pad),
                                                  ptr(R) if with_R else None, ptr(eR) if with_e else None, acc, None, 0,
                                                  st), "tet")
                    assert bool((pad[P.nnz:] == 0.5).all()) and bool((R[P.ndof:] == 0.25).all())
                    out.append((pad, R, eR))
                for a, b in zip(*out):
                    assert float((a - b).abs().max()) <= TOL * max(1.0, float(a.abs().max()))


def tangent80(X, el, u, mu, kappa):
    """Element tangents [E, 12, 12] in 80-bit arithmetic."""
    T = np.longdouble
    d = np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], T)

    def inv(m):
        c = np.stack([np.cross(m[:, 1], m[:, 2]), np.cross(m[:, 2], m[:, 0]), np.cross(m[:, 0], m[:, 1])], 2)
        det = (m[:, 0] * c[:, :, 0]).sum(1)
        return c / det[:, None, None], det
    iJ, det = inv(np.einsum("bm,ebi->eim", d, X.astype(T)[el]))
    g = np.einsum("bm,emi->ebi", d, iJ)
    F = np.eye(3, dtype=T) + np.einsum("ebk,ebi->eki", u.astype(T)[el], g)
    iF, J = inv(F)
    c = mu * np.exp(-2 * np.log(J) / 3)
    I1m = c * (F * F).sum((1, 2))
    q, f = np.einsum("eik,ebi->ebk", iF, g), np.einsum("eki,ebi->ebk", F, g)
    mul = lambda s, a, b, o: np.einsum("e,eaj,ebk->" + o, s * det / 6, a, b)  # noqa: E731
    K = mul(-2 * c / 3, f, q, "eajbk") + mul(-2 * c / 3, q, f, "eajbk")
    K += mul(kappa * J * (2 * J - 1) + 2 * I1m / 9, q, q, "eajbk") + mul(I1m / 3 - kappa * J * (J - 1), q, q, "eakbj")
    K += np.einsum("e,eai,ebi,jk->eajbk", c * det / 6, g, g, np.eye(3, dtype=T))
    return K.reshape(len(el), 12, 12)


@gpu
@pytest.mark.parametrize("dims", [(5, 4, 3), (9, 8, 7)])
def test_tangent_error_is_that_of_the_rank_rounds(dims):
    """Against the element tangents in 80 bits, K by lists is no further off
    than K in rank rounds (2.6e-16 relative, of which the last bits of the
    sums alone make 2 percent either way; 1/J by a cube in place of a division 11 to
    16 percent more)."""
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    X, el = mesh(dims)
    P = DevicePlan(X, np.full(len(X), 7, np.uint8), [("C3D4", el)])
    g = P.groups[0]
    u = np.random.default_rng(4).normal(0, 0.02 / max(dims), X.shape)
    dof = (3 * el[:, :, None] + np.arange(3)).reshape(len(el), 12)
    n = P.ndof
    ip, ix = P.indptr.cpu().numpy(), P.indices.cpu().numpy()
    key = np.repeat(np.arange(n), np.diff(ip)) * n + ix
    ref = np.zeros(P.nnz, np.longdouble)
    np.add.at(ref, np.searchsorted(key, dof[:, :, None] * n + dof[:, None, :]), tangent80(X, el, u, 1.0, 20.0))
    assert P.tangent_lists(0)[0].clist_dev
    old = L.Group()
    C.memmove(C.byref(old), C.byref(g.desc), C.sizeof(L.Group))
    old.clist_dev = None
    gc = torch.from_numpy(u.reshape(-1)).cuda()
    err = []
    for d in (old, g.desc):
        K = torch.empty(P.nnz, dtype=torch.float64, device="cuda")
        L.check(L.fea_assemble_volume(C.byref(P.nodes), C.byref(d), 1.0, 20.0, ptr(gc), ptr(K), None, None, 0, None, 0,
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream)), "tet")
        e = K.cpu().numpy().astype(np.longdouble) - ref
        err.append(float(np.sqrt((e * e).sum() / (ref * ref).sum())))
    assert 1e-17 < err[0] < 1e-15 and err[1] <= 1.04 * err[0], err


def test_lists_of_the_host_plan():
    """Every column's list holds, in incidence order, the blocks of the
    incident elements that fall on its node."""
    from fea_b200 import _lib as L
    from fea_b200.plan import HostPlan
    X, el = mesh((3, 2, 2))
    el[0, 3] = el[0, 2]                           # an element that repeats a node (its values are 0/0)
    N = len(X)
    mask = np.full(N, 7, np.uint8)
    mask[3], mask[5], mask[8] = 0, 6, 1
    hp = HostPlan(N, mask, [(L.FEA_C3D4, el)], [])
    crec, cptr = hp.array(L.FEA_A_G_CREC), hp.array(L.FEA_A_G_CRECPTR)
    clist, nodeinc, inc = hp.array(L.FEA_A_G_CLIST), hp.array(L.G_BASE + L.A_NODEINC), hp.array(L.G_BASE + L.A_INC)
    adjptr, adjcol, adjoff = hp.array(L.FEA_A_ADJPTR), hp.array(L.FEA_A_ADJCOL), hp.array(L.FEA_A_ADJOFF)
    for n in range(N):
        if mask[n] == 0:
            continue
        nb = [n] + [c for c in adjcol[adjptr[n]:adjptr[n + 1]] if c != n]
        assert cptr[n + 1] - cptr[n] == len(nb)
        for u, c in enumerate(nb):
            want = [39 * r + 9 * b for r, q in enumerate(range(nodeinc[n], nodeinc[n + 1]))
                    for b in range(4) if el[inc[q] >> 4, b] == c]
            x, y = (int(v) for v in crec[2 * (cptr[n] + u):2 * (cptr[n] + u) + 2])
            p = adjptr[n] + list(adjcol[adjptr[n]:adjptr[n + 1]]).index(c)
            assert (x & 0xffff, x >> 16) == (adjoff[p], mask[c])
            s, k = y & 0x7ff, y >> 11
            assert list(clist[4 * nodeinc[n] + s:4 * nodeinc[n] + s + k]) == want
    # tiles of at most 128 incidences
    cl, tp = hp.array(L.G_BASE + L.A_CHUNKLIST), hp.array(L.FEA_A_G_TILEPTR)
    assert tp[0] == 0 and tp[-1] == len(cl) and np.all(np.diff(tp) > 0) and len(tp) > 3
    assert np.all(np.diff([nodeinc[n] for n in cl[tp[:-1]]] + [nodeinc[-1]]) <= 128)


@gpu
@pytest.mark.parametrize("kind", [(1, 1, 1), (3, 2, 2), (9, 8, 7), "fan", "mixed"])
def test_lists_made_on_the_device(kind):
    """The device's lists are the host plan's: nodes of 1 to 120 elements and up
    to 122 neighbours, partly and wholly fixed ones, nodes that also belong to
    C3D8 elements or to no element."""
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    from fea_b200.meshes import hex_block
    rng = np.random.default_rng(6)
    X, el = mesh((5, 4, 3) if kind == "mixed" else kind)
    groups = [("C3D4", el)]
    if kind == "mixed":
        groups.insert(0, ("C3D8", rng.permutation(len(X))[hex_block(0, dims=(4, 3, 3))[1]]))
        X, el = np.concatenate([X, rng.uniform(size=(3, 3))]), el[::2]
        groups[1] = ("C3D4", el)
    mask = rng.choice(np.array([7, 7, 7, 7, 5, 2, 0], np.uint8), len(X))
    P = DevicePlan(X, mask, groups)
    gi = len(groups) - 1
    g = P.groups[gi]
    assert g.lists is None and not g.desc.clist_dev           # (made when asked for)
    want = [P.host.array(a, gi) for a in (L.FEA_A_G_CLIST, L.FEA_A_G_CREC)]
    assert (want[0].size, want[1].size) == (4 * g.ninc, 2 * g.nrec)
    out = [torch.full((w.size + 16,), -7, dtype=t, device="cuda") for w, t in zip(want, (torch.int16, torch.int32))]
    L.check(L.fea_tet_lists(C.byref(P.nodes), C.byref(g.desc), ptr(out[0]), ptr(out[1]),
                            C.c_void_p(torch.cuda.current_stream().cuda_stream)), "lists")
    for w, o in zip(want, out):
        assert np.array_equal(o[:-16].cpu().numpy().view(w.dtype), w) and bool((o[-16:] == -7).all())
    d, _ = P.tangent_lists(gi)
    assert d is g.desc and torch.equal(g.lists[0], out[0][:-16]) and torch.equal(g.lists[1], out[1][:-16])


@gpu
@pytest.mark.parametrize("first", ["capture", "warm", "stream", "threads"])
def test_first_tangent(first):
    """The lists come with the first tangent: under capture (whose replays make
    their own), before one, on another stream, from several threads at once; a
    later tangent elsewhere has the same bits."""
    import threading
    from fea_b200 import DevicePlan
    X, el = mesh((9, 8, 7))
    P, Q = (DevicePlan(X, np.full(len(X), 7, np.uint8), [("C3D4", el)]) for _ in range(2))
    gc = torch.from_numpy(np.random.default_rng(2).normal(0, 1e-3, P.ndof)).cuda()

    def tangent(p, K):
        p.assemble_volume(0, 1.0, 30.0, gc, K=K)
        return K
    ref = tangent(Q, P.zeros(P.nnz))
    Ks = [P.zeros(P.nnz) for _ in range(4)]
    torch.cuda.synchronize()
    if first == "capture":
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            tangent(P, Ks[0])
        assert P.groups[0].lists is None
        tangent(P, Ks[1])                         # before the first replay
        for _ in range(2):
            Ks[0].zero_()
            g.replay()
    elif first == "warm":
        tangent(P, Ks[1])
        torch.cuda.synchronize()
        tangent(P, Ks[1])
        assert P.groups[0].lists_done             # the capture takes the plan's lists
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            tangent(P, Ks[0])
        g.replay()
    elif first == "stream":
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            tangent(P, Ks[0])
        tangent(P, Ks[1])
    else:
        def go(k):
            with torch.cuda.stream(torch.cuda.Stream()):
                tangent(P, Ks[k])
                torch.cuda.current_stream().synchronize()
        th = [threading.Thread(target=go, args=(k,)) for k in range(4)]
        [t.start() for t in th]
        [t.join() for t in th]
    torch.cuda.synchronize()
    for k in range(4 if first == "threads" else 2):
        assert torch.equal(Ks[k], ref)


@gpu
@pytest.mark.parametrize("kind", [(1, 1, 1), (2, 1, 1), (11, 1, 2), (9, 8, 7), "fan"])
@pytest.mark.parametrize("fp32", [0, 1])
def test_explicit_steps(kind, fp32):
    """A start and five steps: the short work buffer (every node evaluates its
    elements) and the long one (each element once; counts around the 32 of a
    warp and the 128 of a block)."""
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    X, el = mesh(kind)
    N = len(X)
    mask = np.full(N, 7, np.uint8)
    mask[N // 2], mask[N // 3], mask[-1] = 0, 5, 2
    P = DevicePlan(X, mask, [("C3D4", el)])
    g = P.groups[0]
    h = 1 if kind == "fan" else 1 / max(kind)
    gc = torch.from_numpy(np.random.default_rng(2).normal(0, 5e-3 * h, P.ndof)).cuda()
    v0 = 1e-2 * torch.randn(P.ndof, dtype=torch.float64, generator=torch.Generator().manual_seed(5)).cuda()
    minv = P.lumped_mass_inv([1.0])
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    short = int(L.fea_explicit_work_len(C.byref(P.nodes)))
    n = int(L.fea_explicit_group_work_len(C.byref(P.nodes), C.byref(g.desc)))
    assert n == short + 9 * g.ne
    out = []
    for wn in (short, n):
        pad = torch.full((wn + 64,), 7.25, dtype=torch.float64, device="cuda")
        u, v, vh, a = gc.clone(), v0.clone(), torch.empty_like(gc), torch.empty_like(gc)
        for init, steps in ((1, 2), (0, 3)):
            L.check(L.fea_explicit_run(C.byref(P.nodes), C.byref(g.desc), 1.0, 30.0, ptr(minv), 2e-3 * h, steps, fp32,
                                       init, ptr(u), ptr(vh), ptr(a), ptr(v), ptr(pad), wn, st), "explicit")
        assert bool((pad[wn:] == 7.25).all())
        out.append((u, v, a))
    # FP64: the paths order the products of an element differently (1e-15 of its stresses' terms, which cancel by up
    # to a factor of a hundred).  FP32: kappa * 6e-8 of the stresses' scale, which the strains' 1e-2 magnifies
    tol = 2e-3 if fp32 else TOL * 10
    for x, y in zip(*out):
        assert float((x - y).abs().max()) <= tol * float(x.abs().max())
