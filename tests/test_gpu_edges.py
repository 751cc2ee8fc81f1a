"""The kernels at the sizes and layouts where they can go wrong: tile edges and
remainders, unaligned buffers, unsorted and repeated observations."""
import dataclasses

import numpy as np
import pytest

import oracle
from conftest import block_rel_err
from uncertaintyte_b200 import native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", range(1, 10))
def test_block_eigen_of_every_size_and_scale(dim):
    """Sub-blocks of 9 x 9 blocks (37 of them: partial warps), at scales whose squares leave the
    FP64 range (rotations by the tangent); the accessors' 1e-12, and 1e-12 of their scale."""
    rng = np.random.default_rng(dim)
    X = rng.standard_normal((37, 9, 9))
    A = np.einsum("bij,bkj->bik", X, X) * np.array([1e-145, 1.0, 1e145])[np.arange(37) % 3, None, None]
    iu = np.triu_indices(9)
    off = (9 - dim) // 2
    vals, vecs = native.block_eigen(A[:, iu[0], iu[1]].reshape(-1), 9, sub_offset=off, sub_dim=dim)
    B = A[:, off:off + dim, off:off + dim]
    ref = np.linalg.eigvalsh(B)[:, ::-1]
    scale = np.abs(ref).max(axis=1)
    assert np.max(np.abs(vals - ref) / scale[:, None]) < 1e-12
    V = np.transpose(vecs, (0, 2, 1))
    res = np.einsum("bij,bjk->bik", B, V) - V * vals[:, None, :]
    assert np.max(np.abs(res) / scale[:, None, None]) < 1e-12
    assert np.max(np.abs(np.einsum("bji,bjk->bik", V, V) - np.eye(dim))) < 1e-12


@pytest.mark.parametrize("n", [1, 31, 64, 127, 130, 257])
def test_jacobian_remainders_and_unaligned_outputs(n):
    """Any number of observations, outputs 4 (columns) and 8 (values) bytes past a 16-byte boundary:
    the same bytes as the whole scene's, and nothing written past the end."""
    import torch
    sc = scenes.make_sized_scene(12, 40, 3, seed=4)
    dev = "cuda"
    cams, pts = torch.from_numpy(sc.cams.copy()).to(dev), torch.from_numpy(sc.points.copy()).to(dev)
    oc, op = torch.from_numpy(sc.obs_cam.copy()).to(dev), torch.from_numpy(sc.obs_pt.copy()).to(dev)

    def run(count, shift):
        rows = torch.zeros(2 * count + 1, dtype=torch.int32, device=dev)
        cols = torch.full((24 * count + 8,), -7, dtype=torch.int32, device=dev)
        vals = torch.full((24 * count + 8,), -7.0, dtype=torch.float64, device=dev)
        native._check(native.lib().unc_jacobian_device(
            len(sc.cams), len(sc.points), count, cams.data_ptr(), pts.data_ptr(), oc.data_ptr(), op.data_ptr(),
            rows.data_ptr(), cols.data_ptr() + 4 * shift, vals.data_ptr() + 8 * shift, None))
        torch.cuda.synchronize()
        return rows.cpu(), cols[shift:].cpu(), vals[shift:].cpu()

    rows, cols, vals = run(len(sc.obs_cam), 0)
    for shift in (0, 1):
        r, c, v = run(n, shift)
        assert torch.equal(r, rows[:2 * n + 1])
        assert torch.equal(c[:24 * n], cols[:24 * n]) and torch.equal(v[:24 * n], vals[:24 * n])
        assert (c[24 * n:] == -7).all() and (v[24 * n:] == -7.0).all()


@pytest.mark.parametrize("m,n,k", [(33, 31, 1), (63, 65, 15), (65, 64, 17), (96, 32, 47), (766, 768, 65),
                                   (832, 830, 63), (2112, 15, 130)])
def test_gemm_f64_tile_edges(m, n, k):
    """Either side of the 32 x 32 and 64 x 64 tiles, of their stages of 16 k and of the tile count at
    which the small tile gives way; k products and the result rounded: k eps of the largest sum."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + 3 * n + k)
    lda, ldb, ldc = m + (m & 1), k + (k & 1), m + (m & 1) + 2
    A = torch.randn((k, lda), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((n, ldb), dtype=torch.float64, device="cuda", generator=g)
    C = torch.full((n, ldc), 3.0, dtype=torch.float64, device="cuda")
    native.gemm_f64_device(m, n, k, 1.0, A.data_ptr(), lda, B.data_ptr(), ldb, 0.0, C.data_ptr(), ldc)
    torch.cuda.synchronize()
    ref = (A[:, :m].T @ B[:, :k].T).T
    bound = k * 2.2e-16 * (A[:, :m].abs().T @ B[:, :k].abs().T).max().item()
    assert (C[:, :m] - ref).abs().max().item() <= bound
    assert (C[:, m:] == 3.0).all()


@pytest.mark.parametrize("n,ld", [(129, 131), (64, 65), (257, 258)])
def test_mixed_product_of_any_leading_dimension(n, ld):
    """Rows that start off the 16-byte boundaries are sliced and written by single elements: the
    same bytes as aligned ones."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    P, X = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    out = []
    for pitch in (ld, (n + 7) // 8 * 8):
        p, x, c = (torch.zeros((n, pitch), dtype=torch.float64, device="cuda") for _ in range(3))
        p[:, :n], x[:, :n] = P, X
        native.gemm_mixed_device(n, p.data_ptr(), x.data_ptr(), pitch, c.data_ptr(), 5)
        torch.cuda.synchronize()
        assert (c[:, n:] == 0).all()
        out.append(c[:, :n].clone())
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("power", [-900, 0, 900])
def test_mixed_product_of_scaled_and_zero_rows(power):
    """A row's exponent is that of its largest entry: operands scaled by a power of two give the same
    digits, so exactly the scaled result, and rows of zeros give zeros."""
    import torch
    n = 200
    g = torch.Generator(device="cuda").manual_seed(7)
    P = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    X = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    P, X = P + P.T, X + X.T
    P[17], P[:, 17] = 0.0, 0.0
    out = []
    for scale in (1.0, 2.0 ** power):
        p, c = P * scale, torch.full((n, n), 5.0, dtype=torch.float64, device="cuda")
        native.gemm_mixed_device(n, p.data_ptr(), X.data_ptr(), n, c.data_ptr(), 5)
        torch.cuda.synchronize()
        out.append(c)
    assert torch.equal(out[0] * 2.0 ** power, out[1])
    assert (out[0][:, 17] == 0).all()


@pytest.mark.parametrize("cams,points,obs", [(5200, 800, 12000), (2, 1, 3000), (40, 1025, 9000)])
def test_index_of_unsorted_observations(cams, points, obs):
    """J^T J of observations in random order, some of them repeated: more cameras than one pass of
    the index takes, and lists of thousands at one point."""
    rng = np.random.default_rng(cams)
    oc, op = rng.integers(0, cams, obs), rng.integers(0, points, obs)
    cols = np.empty((obs, 2, 12), dtype=np.int32)
    cols[:, :, :9] = (9 * oc)[:, None, None] + np.arange(9)
    cols[:, :, 9:] = (9 * cams + 3 * op)[:, None, None] + np.arange(3)
    vals = rng.standard_normal(24 * obs)
    rows = (12 * np.arange(2 * obs + 1)).astype(np.int32)
    num_cols = 9 * cams + 3 * points
    r, c, v = native.jtj_crs(2 * obs, num_cols, rows, cols.reshape(-1), vals, cams)
    ro, co, vo = oracle.jtj(2 * obs, num_cols, rows, cols.reshape(-1), vals)
    np.testing.assert_array_equal(r, ro)
    np.testing.assert_array_equal(c, co)
    np.testing.assert_allclose(v, vo, rtol=0, atol=1e-12 * np.abs(vo).max())


def _from_blocks(sc, order, scale=None):
    """The Jacobian of the observations `order` (indices, repeats allowed), rows scaled."""
    jac = scenes.scene_jacobian(sc)
    cols, vals = jac.cols.reshape(-1, 24)[order], jac.values.reshape(-1, 24)[order].copy()
    if scale is not None:
        vals *= np.asarray(scale)[:, None]
    n = len(order)
    return dataclasses.replace(jac, num_obs=n, num_rows=2 * n, rows=(12 * np.arange(2 * n + 1)).astype(np.int32),
                               cols=cols.reshape(-1).copy(), values=vals.reshape(-1).copy(), lam=1e-5)


@pytest.mark.parametrize("cams,points", [(3, 700), (12, 60), (60, 50)])
def test_schur_of_repeated_and_unsorted_observations(cams, points):
    """A camera that sees a point m times gives m equal terms: the cameras' covariances are those of
    one observation scaled by sqrt(m). m = 1 .. 4, in random order; 3 cameras: columns of several
    chunks. lambda = 1e-5 keeps the condition number near 1e5: 1e-9 is the FP64 bar."""
    rng = np.random.default_rng(cams)
    sc = scenes.make_sized_scene(cams, points, 3, seed=cams)
    m = rng.integers(1, 5, len(sc.obs_cam))
    order = rng.permutation(np.repeat(np.arange(len(m)), m))
    one, _, _ = native.compute_covariances(_from_blocks(sc, np.arange(len(m)), np.sqrt(m)))
    many, _, _ = native.compute_covariances(_from_blocks(sc, order))
    assert block_rel_err(many, one, 45) < 1e-9


def test_points_of_too_many_observations_are_refused():
    sc = scenes.make_sized_scene(6, 20, 3, seed=1)
    at = int(np.flatnonzero(sc.obs_pt == 5)[0])
    with pytest.raises(native.UncError) as e:
        native.compute_covariances(_from_blocks(sc, np.concatenate([np.arange(len(sc.obs_cam)), np.full(12288, at)])))
    assert e.value.status == -8
    native.compute_covariances(_from_blocks(sc, np.arange(len(sc.obs_cam))))


def test_one_context_through_precisions_and_sizes():
    """A context that changes precision, size and output kind gives each call the bytes of a fresh
    context (captured inverses are not replayed for another call's buffers)."""
    calls = [("small", "mixed"), ("small", "fp64"), ("medium", "mixed"), ("small", "mixed"), ("medium", "fp64"),
             ("medium", "mixed")]
    jacs = {name: scenes.synthetic_jacobian(name, seed=1) for name in ("small", "medium")}
    fresh = {}
    for key in set(calls):
        with native.Context(0) as c:
            fresh[key] = native.compute_covariances(jacs[key[0]], c, precision=key[1])[:2]
    with native.Context(0) as c:
        for key in calls:
            cam, pt, _ = native.compute_covariances(jacs[key[0]], c, precision=key[1])
            np.testing.assert_array_equal(cam, fresh[key][0])
            np.testing.assert_array_equal(pt, fresh[key][1])
