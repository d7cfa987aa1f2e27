"""C3D8 kernels that evaluate each element once (slots per element and node,
then a sum per node) against the general path (every node evaluates its
elements), which the same entry points take without the slots' buffer.

Meshes: element counts around the 16 of a CTA, one element, constrained
components, shuffled node numbers, an element that repeats a node.  Both
paths sum at most 8 elements x 8 Gauss points per entry with relative error
of a few 1e-15 per term; entries cancel by up to a factor of a hundred in the
near-incompressible residual: 1e-12 of the largest entry bounds the
difference."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import fea_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-12
MESHES = [(1, 1, 1), (5, 3, 1), (4, 2, 2), (17, 1, 1), (3, 4, 5)]


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def hex_plan(dims, shuffle=True, repeat=False, seed=3):
    """Plan of a jittered block with a clamped node and a partly fixed one,
    and a displacement; repeat: one element uses a node twice."""
    from fea_b200 import DevicePlan
    from fea_b200.meshes import hex_block
    rng = np.random.default_rng(seed)
    X, el = hex_block(0, jitter=0.1, seed=seed, dims=dims)
    N = X.shape[0]
    if shuffle:
        perm = rng.permutation(N)
        inv = np.empty(N, np.int64)
        inv[perm] = np.arange(N)
        X, el = X[perm], inv[el]
    if repeat:                                    # a wedge: edge 4-7 of the last element collapsed onto node 4
        el = el.copy()
        el[-1, 7] = el[-1, 4]
    mask = np.full(N, 7, np.uint8)
    mask[0], mask[N // 2] = 0, 5
    P = DevicePlan(X, mask, [("C3D8", el)])
    h = 1.0 / max(dims)
    gc = torch.from_numpy(rng.normal(0, 0.02 * h, P.ndof)).cuda()
    return P, gc


def close(a, b):
    s = float(b.abs().max())
    return float((a - b).abs().max()) <= TOL * s


@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("acc", [0, 1])
@pytest.mark.parametrize("repeat", [False, True])
def test_residual(dims, acc, repeat):
    from fea_b200 import _lib as L
    P, gc = hex_plan(dims, repeat=repeat)
    g = P.groups[0]
    n = int(L.fea_force_work_len(C.byref(g.desc)))
    assert n == g.ne * 32
    pad = torch.full((n + 64,), 7.25, dtype=torch.float64, device="cuda")
    base = torch.linspace(-1, 1, P.ndof, dtype=torch.float64, device="cuda")
    out = []
    for w, wn in ((None, 0), (pad, n - 1), (pad, n)):
        R, eR = base.clone(), torch.zeros(24 * g.ne, dtype=torch.float64, device="cuda")
        L.check(L.fea_assemble_volume(C.byref(P.nodes), C.byref(g.desc), 1.0, 40.0, ptr(gc), None, ptr(R), ptr(eR), acc,
                                      ptr(w), wn, stream()), "force")
        out.append((R - base if acc else R, eR))
        if wn < n:                                # too short a buffer is left alone
            assert bool((pad == 7.25).all())
    assert bool((pad[n:] == 7.25).all())
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert close(out[2][1], out[0][1])            # element residuals
    if acc:                                       # (the sums are rounded to the base's size)
        assert float((out[2][0] - out[0][0]).abs().max()) <= TOL * max(1.0, float(out[0][0].abs().max()))
    else:
        assert close(out[2][0], out[0][0])


def test_residual_on_streams_and_under_capture():
    """Every call takes its slots from the allocator of its stream or of the
    capture, with the same bits."""
    P, gc = hex_plan((6, 5, 4))
    ref = P.zeros(P.ndof)
    P.assemble_volume(0, 1.0, 40.0, gc, R=ref)
    torch.cuda.synchronize()
    side, outs = torch.cuda.Stream(), []
    side.wait_stream(torch.cuda.current_stream())
    for k in range(8):                            # interleaved launches on two streams
        a, b = P.zeros(P.ndof), P.zeros(P.ndof)
        side.wait_stream(torch.cuda.current_stream())
        P.assemble_volume(0, 1.0, 40.0, gc, R=a)
        with torch.cuda.stream(side):
            P.assemble_volume(0, 1.0, 40.0, gc, R=b)
        outs += [a, b]
    torch.cuda.synchronize()
    assert all(torch.equal(o, ref) for o in outs)
    R = P.zeros(P.ndof)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        P.assemble_volume(0, 1.0, 40.0, gc, R=R)
    R.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(R, ref)


def test_residual_matches_the_oracle():
    X, el = O.hex_block(3, jitter=0.1, seed=2)
    from fea_b200 import DevicePlan
    N = X.shape[0]
    P = DevicePlan(X, np.full(N, 7, np.uint8), [("C3D8", el.numpy())])
    gc = 1e-2 * torch.randn(3 * N, generator=torch.Generator().manual_seed(1), dtype=torch.float64)
    R = P.zeros(P.ndof)
    P.assemble_volume(0, 1.0, 40.0, gc.cuda(), R=R)
    m = O.Model(X, [O.Group("C3D8", el, 1.0, 40.0)], [], [])
    assert close(R.cpu(), m.assemble(gc, want_K=False)[0])


@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("repeat", [False, True])
def test_vjp(dims, repeat):
    from fea_b200 import _lib as L
    P, gc = hex_plan(dims, repeat=repeat)
    g = P.groups[0]
    n = int(L.fea_adjoint_work_len(C.byref(g.desc)))
    lam = torch.randn(P.n_nodes, 3, dtype=torch.float64, generator=torch.Generator().manual_seed(4)).cuda()
    pad = torch.full((n + 64,), 7.25, dtype=torch.float64, device="cuda")
    short = int(L.fea_reduce_scratch_len(g.ne))
    out = []
    for wn in (short, n):
        dX = torch.zeros(P.n_nodes, 3, dtype=torch.float64, device="cuda")
        dmu = torch.zeros(1, dtype=torch.float64, device="cuda")
        L.check(L.fea_adjoint_vjp_volume(C.byref(P.nodes), C.byref(g.desc), 1.0, 40.0, ptr(gc), ptr(lam), ptr(dX),
                                         ptr(dmu), ptr(pad), wn, stream()), "vjp")
        assert bool((pad[wn:] == 7.25).all())
        out.append((dX, dmu))
    assert close(out[1][0], out[0][0])
    # a sum of 8 ne signed terms: against the sum of their sizes' bound
    assert abs(float(out[1][1] - out[0][1])) <= TOL * max(float(out[0][1].abs()), g.ne * 1e-2)


@pytest.mark.parametrize("dims", MESHES)
@pytest.mark.parametrize("fp32", [0, 1])
def test_explicit_steps(dims, fp32):
    """A start and five steps: the C ABI with the short work buffer (the
    per-node path) and with the slots."""
    from fea_b200 import _lib as L
    P, gc = hex_plan(dims)
    g = P.groups[0]
    minv = P.lumped_mass_inv([1.0])
    short = int(L.fea_explicit_work_len(C.byref(P.nodes)))
    n = int(L.fea_explicit_group_work_len(C.byref(P.nodes), C.byref(g.desc)))
    assert n == short + 32 * g.ne
    v0 = 0.01 * torch.randn(P.ndof, dtype=torch.float64, generator=torch.Generator().manual_seed(5)).cuda()
    dt = 0.02 / max(dims)
    out = []
    for wn in (short, n):
        pad = torch.full((wn + 64,), 7.25, dtype=torch.float64, device="cuda")
        u, v, vh, a = gc.clone(), v0.clone(), torch.empty_like(gc), torch.empty_like(gc)
        for init, steps in ((1, 2), (0, 3)):
            L.check(L.fea_explicit_run(C.byref(P.nodes), C.byref(g.desc), 1.0, 40.0, ptr(minv), dt, steps, fp32, init,
                                       ptr(u), ptr(vh), ptr(a), ptr(v), ptr(pad), wn, stream()), "explicit")
        assert bool((pad[wn:] == 7.25).all())
        out.append((u, v, a))
    # FP32 element math: the accelerations' error is kappa * 6e-8 of the stresses' scale per Gauss point
    # (3e-5 of the largest acceleration, either path)
    tol = 1e-4 if fp32 else TOL * 10
    for x, y in zip(*out):
        assert float((x - y).abs().max()) <= tol * float(x.abs().max())


def test_plans_hold_no_slots(monkeypatch):
    """The slots live for one call: neither a new plan nor one that has
    computed residuals and gradients holds them, and without memory for them
    the general path gives the same."""
    from fea_b200 import DevicePlan
    from fea_b200.meshes import hex_block
    X, el = hex_block(0, dims=(24, 24, 24))

    def plan():
        return DevicePlan(X, np.full(len(X), 7, np.uint8), [("C3D8", el)])
    def used():                                   # (what was asked for, not the blocks it got)
        return torch.cuda.memory_stats()["requested_bytes.all.current"]
    P = plan()
    before = used()
    Q = plan()
    held = used() - before
    arrays = sum(t.numel() * t.element_size() for o in (Q, Q.groups[0]) for t in vars(o).values() if isinstance(t, torch.Tensor))
    slots = 8 * 32 * len(el)
    assert 0.9 * arrays < held < arrays + slots / 4
    gc = 1e-3 * torch.randn(P.ndof, dtype=torch.float64, generator=torch.Generator().manual_seed(5)).cuda()
    lam = torch.randn(P.n_nodes, 3, dtype=torch.float64, generator=torch.Generator().manual_seed(4)).cuda()
    out, empty = [], torch.empty

    def no_room(n, *a, **k):
        if n >= slots / 8:
            raise torch.cuda.OutOfMemoryError("no room for %d" % n)
        return empty(n, *a, **k)
    for tight in (True, False):
        R, dX, dmu = P.zeros(P.ndof), torch.zeros_like(lam), P.zeros(1)
        before = used()
        with monkeypatch.context() as m:
            if tight:
                m.setattr(torch, "empty", no_room)
            P.assemble_volume(0, 1.0, 40.0, gc, R=R)
            P.adjoint_vjp_volume(0, 1.0, 40.0, gc, lam, dX, dmu)
        assert used() - before < slots / 4
        out.append((R, dX))
    assert not torch.equal(*[o[0] for o in out])  # two paths, to rounding the same
    for x, y in zip(*out):
        assert close(x, y)


@pytest.mark.parametrize("kind", ["C3D8", "C3D4"])
def test_explicit_run_where_the_long_buffer_does_not_fit(kind, monkeypatch):
    """Without memory for the elements' parts DevicePlan.explicit_run takes the
    per-node path, as it did before it had another."""
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    from fea_b200.meshes import hex_block, tet_block
    X, el = (hex_block if kind == "C3D8" else tet_block)(0, dims=(9, 8, 7))
    P = DevicePlan(X, np.full(len(X), 7, np.uint8), [(kind, el)])
    u0 = 1e-3 * torch.randn(P.ndof, dtype=torch.float64, generator=torch.Generator().manual_seed(5)).cuda()
    minv = P.lumped_mass_inv([1.0])
    short = int(L.fea_explicit_work_len(C.byref(P.nodes)))
    assert int(L.fea_explicit_group_work_len(C.byref(P.nodes), C.byref(P.groups[0].desc))) > short > P.ndof
    empty = torch.empty

    def no_room(n, *a, **k):
        if n > short:
            raise torch.cuda.OutOfMemoryError("no room for %d" % n)
        return empty(n, *a, **k)
    out = []
    for tight in (True, False):                   # (first without room: nothing may be kept from an earlier call)
        u, v = u0.clone(), torch.zeros_like(u0)
        vh, a = torch.zeros_like(u0), torch.zeros_like(u0)
        with monkeypatch.context() as m:
            if tight:
                m.setattr(torch, "empty", no_room)
            P.explicit_run(0, 1.0, 40.0, minv, 1e-3, 4, u, vh, a, v, init=True)
        out.append((u, v, a))
    for x, y in zip(*out):
        assert not torch.equal(x, u0) and float((x - y).abs().max()) <= 10 * TOL * float(x.abs().max())


@pytest.mark.parametrize("dims", MESHES + [(13, 8, 11), (12, 11, 12), (14, 13, 13)])
@pytest.mark.parametrize("repeat", [False, True])
def test_tangent_and_residual(dims, repeat):
    """One, two (1,185 elements and more) and four (2,369 and more) elements
    per warp, with accumulate and the element residual."""
    P, gc = hex_plan(dims, repeat=repeat)
    g, N = P.groups[0], P.n_nodes
    X, el = P.X.cpu().view(N, 3), g.conn.cpu().view(-1, 8).long()
    m = O.Model(X, [O.Group("C3D8", el, 1.0, 40.0)], [], [])
    m._free = (P.mask.cpu().view(N, 1) >> torch.arange(3) & 1).bool().reshape(-1)
    used = torch.zeros(N, 3, dtype=torch.bool)    # a node of no element keeps what R held
    used[el] = True
    used = used.reshape(-1)[m.free_mask()]
    R0, (ip, ix, K0) = m.assemble(gc.cpu())
    assert torch.equal(P.indices.cpu().long(), ix.long())
    e0 = O.element_residual_tangent("C3D8", X, el, m.gc_to_u(gc.cpu()), 1.0, 40.0, False)[0]
    for acc in (False, True):
        K, R = torch.full((P.nnz,), 0.5, dtype=torch.float64, device="cuda"), torch.full_like(gc, 0.25)
        eR = torch.zeros(24 * g.ne, dtype=torch.float64, device="cuda")
        P.assemble_volume(0, 1.0, 40.0, gc, K=K, R=R, elemR=eR, accumulate=acc)
        assert float((K.cpu() - (0.5 if acc else 0.0) - K0).abs().max()) <= TOL * float(K0.abs().max())
        d = (R.cpu() - (0.25 if acc else 0.0) - R0)[used]
        assert float(d.abs().max()) <= TOL * max(1.0, float(R0.abs().max()))
        assert close(eR.cpu(), e0.reshape(-1))
        K2 = torch.full_like(K, 0.5)
        P.assemble_volume(0, 1.0, 40.0, gc, K=K2, accumulate=acc)
        assert torch.equal(K, K2)
