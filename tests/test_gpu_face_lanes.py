"""Follower pressure with 4 lanes per (node, face) (k_face_rk4, chunks of 32
incidences) against the thread-per-incidence kernel, which the entry point
takes for a plan whose chunks hold 128: Q4 and T3 surfaces, shuffled nodes,
partly fixed ones, K or R alone, added to values that are there.  Each entry
is a sum of a few faces' Gauss points: 1e-13 of the largest."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("kind,face", [("C3D8", "Q4"), ("C3D4", "T3")])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 2), (3, 7, 6), (2, 17, 9)])
def test_matches_thread_per_incidence(kind, face, dims):
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    from fea_b200.meshes import hex_block, plane_faces, tet_block
    rng = np.random.default_rng(3)
    X, el = (hex_block if kind == "C3D8" else tet_block)(0, dims=dims)
    X = X + 1.0                                   # the faces' planes off the origin
    _, faces = plane_faces(kind, el, X, 0, 2.0)
    N = len(X)
    X = X + rng.uniform(-0.05, 0.05, X.shape) / max(dims)
    perm = rng.permutation(N)
    inv = np.empty(N, np.int64)
    inv[perm] = np.arange(N)
    X, el, faces = X[perm], inv[el], inv[faces]
    mask = np.full(N, 7, np.uint8)
    mask[faces[0, 0]], mask[faces[-1, 1]], mask[faces[0, 2]] = 5, 0, 2
    P = DevicePlan(X, mask, [(kind, el)], [(face, faces)])
    f = P.faces[0]
    assert f.desc.threads == 32
    Xi = torch.from_numpy(X).cuda()
    gc = torch.from_numpy(rng.normal(0, 0.01 / max(dims), P.ndof)).cuda()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    # the other kernel on the same chunks: a CTA of 128 threads holds 32 incidences too
    old = L.Group()
    C.memmove(C.byref(old), C.byref(f.desc), C.sizeof(L.Group))
    old.threads = 128
    for with_K, with_R in ((True, True), (True, False), (False, True)):
        out = []
        for d in (old, f.desc):
            K = torch.linspace(-1, 1, P.nnz + 32, dtype=torch.float64, device="cuda")
            R = torch.linspace(-1, 1, P.ndof + 32, dtype=torch.float64, device="cuda")
            L.check(L.fea_assemble_pressure(C.byref(P.nodes), C.byref(d), 0.7, ptr(Xi), ptr(gc),
                                            ptr(K) if with_K else None, ptr(R) if with_R else None, st), "pressure")
            out.append((K, R))
        for a, b in zip(*out):
            assert float((a - b).abs().max()) <= 1e-13 * max(1.0, float(a.abs().max()))
        base = torch.linspace(-1, 1, P.nnz + 32, dtype=torch.float64, device="cuda")
        assert with_K == (not torch.equal(out[1][0], base))


@pytest.mark.parametrize("dims", [(2, 1, 1), (2, 3, 2), (2, 9, 7)])
def test_faces_that_repeat_a_node(dims):
    """Q4 faces with one collapsed edge (every edge in turn, and a whole
    surface of them): two lanes of an incidence then hold the same columns.
    Against the thread-per-incidence kernel and the CPU oracle, K alone and K
    with R, the same bits from run to run."""
    from fea_b200 import DevicePlan
    from fea_b200 import _lib as L
    from fea_b200.meshes import hex_block, plane_faces
    from oracle import fea_oracle as O
    rng = np.random.default_rng(5)
    X, el = hex_block(0, dims=dims)
    X = X + 1.0
    _, faces = plane_faces("C3D8", el, X, 0, 2.0)
    X = X + rng.uniform(-0.05, 0.05, X.shape) / max(dims)
    faces = faces.copy()
    for i in range(len(faces)):                   # one node of an edge takes the place of the other
        faces[i, (i + 1) % 4] = faces[i, i % 4]
    perm = rng.permutation(len(X))
    inv = np.empty(len(X), np.int64)
    inv[perm] = np.arange(len(X))
    X, el, faces = X[perm], inv[el], inv[faces]
    mask = np.full(len(X), 7, np.uint8)
    if len(faces) > 1:
        mask[faces[0, 2]], mask[faces[-1, 0]] = 5, 0
    P = DevicePlan(X, mask, [("C3D8", el)], [("Q4", faces)])
    f = P.faces[0]
    assert f.desc.threads == 32
    Xi = torch.from_numpy(X).cuda()
    gc = torch.from_numpy(rng.normal(0, 0.01 / max(dims), P.ndof)).cuda()
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    other = L.Group()
    C.memmove(C.byref(other), C.byref(f.desc), C.sizeof(L.Group))
    other.threads = 128

    def run(d, with_R):
        K, R = P.zeros(P.nnz), P.zeros(P.ndof)
        L.check(L.fea_assemble_pressure(C.byref(P.nodes), C.byref(d), 0.7, ptr(Xi), ptr(gc), ptr(K),
                                        ptr(R) if with_R else None, st), "pressure")
        return K, R
    free = torch.from_numpy(((mask[:, None] >> np.arange(3)) & 1).astype(bool))
    x = torch.from_numpy(X.copy())
    x[free] += gc.cpu()
    Rf, k = O.pressure_force_tangent(x, torch.from_numpy(faces), 0.7)
    fi = torch.from_numpy(3 * faces[:, None, :] + np.arange(3)[None, :, None])          # [F, 3, 4] all-DOF indices
    n3 = 3 * len(X)
    Kd = torch.zeros(n3 * n3, dtype=torch.float64)
    Kd.index_add_(0, (fi[:, :, :, None, None] * n3 + fi[:, None, None, :, :]).reshape(-1), -k.reshape(-1))
    Rd = torch.zeros(n3, dtype=torch.float64).index_add_(0, fi.reshape(-1), -Rf.reshape(-1))
    fr = free.reshape(-1)
    Kd = Kd.view(n3, n3)[fr][:, fr]
    ip, ix = P.indptr.cpu(), P.indices.cpu().long()
    rows = torch.repeat_interleave(torch.arange(P.ndof), ip[1:] - ip[:-1])
    ref = Kd[rows, ix]
    for with_R in (False, True):
        K, R = run(f.desc, with_R)
        Ko, Ro = run(other, with_R)
        for a, b in ((K, Ko), (R, Ro), (K.cpu(), ref), (R.cpu(), Rd[fr] if with_R else torch.zeros(P.ndof, dtype=torch.float64))):
            assert float((a - b).abs().max()) <= 1e-13 * max(1.0, float(b.abs().max()))
        for _ in range(3):
            assert torch.equal(run(f.desc, with_R)[0], K)
