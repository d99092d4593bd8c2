"""The body kernel's Gauss-point pass over tiles at the sizes where its branches change: points of one
support and of more than the head rows a thread holds in registers, groups that are not full, many
more touched nodes than point threads, and tile sizes from the smallest up.  Internal forces of one
step against the oracle, bit for bit in FP64; in the mixed form within the rounding of its FP32
strain, stress and contributions."""
import numpy as np
import pytest

from conftest import flat_of, squeezed_lattice
from test_tiles import thinned

pytestmark = pytest.mark.gpu


def fields(counts):
    flat = thinned(flat_of(squeezed_lattice(3, 3)), 3, counts)
    st = np.zeros((len(flat["node_domain"]), 12))
    deform = np.repeat(np.asarray(flat["body_type"]) == 0, np.diff(flat["body_node_ptr"]))
    st[deform, 6:8] = np.random.default_rng(4).standard_normal((int(deform.sum()), 2)) * 1e-9
    flat["node_state"] = st.reshape(-1)
    return flat


def mixed_reference(flat):
    """Internal forces in FP64 by numpy with the displacements relative to the body's first node, as the
    mixed form takes them (the drawn derivatives do not sum to zero, so that the two differ here), and
    per node the rounding allowed: the sum over its entries of c0 |dN| (2 mu + lambda) sum |dN| |u - u0|,
    times the unit roundoff of FP32 and the number of operations behind a contribution (two per
    support, and ten)."""
    b_of = np.repeat(np.arange(len(flat["body_type"])), np.diff(flat["body_gp_ptr"]))
    cnt = np.diff(flat["gp_sup_ptr"])
    n = len(cnt)
    row = np.repeat(np.arange(n), cnt)
    n0 = np.asarray(flat["body_node_ptr"])[b_of[row]]
    col = np.asarray(flat["gp_sup_idx"]) + n0
    up = flat["node_state"].reshape(-1, 12)[:, 6:8]
    dx, dy, u = flat["gp_dNdx"], flat["gp_dNdy"], up[col] - up[n0]
    mat = np.asarray(flat["material_params"]).reshape(-1, len(flat["material_params"]) // len(flat["material_type"]))
    mu, lam = mat[0, 3], mat[0, 4]
    total = lambda v: np.bincount(row, weights=v, minlength=n)
    e11, e22, e12 = total(dx * u[:, 0]), total(dy * u[:, 1]), 0.5 * total(dx * u[:, 1] + dy * u[:, 0])
    s33 = lam * (e11 + e22)
    s11, s22, s12 = s33 + 2 * mu * e11, s33 + 2 * mu * e22, 2 * mu * e12
    c0 = (flat["gp_weight"] * flat["gp_jacobian"])[row]
    node = lambda v: np.bincount(col, weights=v, minlength=len(up))
    f = -np.stack([node(c0 * (dx * s11[row] + dy * s12[row])), node(c0 * (dy * s22[row] + dx * s12[row]))], axis=1)
    d = np.abs(dx) + np.abs(dy)
    strain = total(d * (np.abs(up[col]).sum(axis=1) + np.abs(up[n0]).sum(axis=1)))
    return f, node(c0 * d * (2 * mu + lam) * strain[row] * (2 * cnt[row] + 10) * 2.0 ** -24)


@pytest.mark.parametrize("counts", [[1], [7, 8, 9], [11, 12, 13], [1, 16, 140], [20, 33]])
@pytest.mark.parametrize("cap", [2048, 3840])
def test_internal_forces(gpu_lib, oracle_built, monkeypatch, counts, cap):
    from melody2d_b200.solver import Solver
    from oracle.pyoracle import Oracle
    flat = fields(counts)
    o = Oracle(flat, correctly_rounded=True)
    o.step(1, proximity=False)
    ref = o.forces()["internal"]
    assert np.abs(ref).max() > 0
    monkeypatch.setenv("MELGPU_CHUNK_CAP", str(cap))
    for precision in (0, 1):
        s = Solver.from_flat(flat, precision=precision)
        assert s.kernel_config()["chunk_cap"] == (max(cap, 4096) if precision else cap)
        s.record_forces()
        s.step(1, proximity=False)
        f = s.forces()["internal"]
        if precision == 0:
            np.testing.assert_array_equal(f, ref)
        else:
            near, bound = mixed_reference(flat)
            assert (np.abs(f - near) <= bound[:, None]).all()
        s.close()
