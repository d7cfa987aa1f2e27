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
