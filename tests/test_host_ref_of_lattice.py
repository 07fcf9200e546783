"""The closed form of the reference's node numbering on the lattice (ref_of_lattice,
csrc/ctx.cuh), restated here and compared with the numbering that the mesh
builder produces edge by edge (first-seen midpoints), for every node."""
import numpy as np
import pytest

from dimspers_b200 import build_mesh


def ref_of_lattice(a, b, ncr, nct):
    ia, jb = a >> 1, b >> 1
    nv = (ncr + 1) * nct

    def base(it):
        return 0 if it == 0 else 4 * ncr + 1 + (it - 1) * (3 * ncr + 1)

    per = 4 if jb == 0 else (2 if jb == nct - 1 else 3)    # midpoints that a cell of this column adds
    if not a & 1 and not b & 1:
        return ia + (ncr + 1) * jb
    if a & 1 and b & 1:
        return nv + base(jb) + per * ia + 1
    if b & 1:
        return nv + base(jb) + per * ia
    if jb == 0:
        return nv + 4 * ia + 2
    it = jb - 1
    return nv + base(it) + (4 * ia + 3 if it == 0 else 3 * ia + 2)


LOC = (((0, 0), (0, 2), (2, 0), (0, 1), (1, 1), (1, 0)), ((0, 2), (2, 2), (2, 0), (1, 2), (2, 1), (1, 1)))


@pytest.mark.parametrize("ncr,nct", [(1, 3), (1, 4), (2, 3), (3, 5), (4, 32), (7, 9), (8, 64), (31, 20), (5, 101)])
def test_closed_form_matches_mesh_builder(ncr, nct):
    mesh = build_mesh(ncr, nct, colors=False)
    seen = np.zeros(mesh.nnod, dtype=bool)
    for q in range(ncr * nct):
        ir, it = q % ncr, q // ncr
        for t in (0, 1):
            for k, (da, db) in enumerate(LOC[t]):
                a, b = 2 * ir + da, (2 * it + db) % (2 * nct)
                n = ref_of_lattice(a, b, ncr, nct)
                assert n == mesh.e2n[k, 2 * q + t]
                seen[n] = True
    assert seen.all()
