"""Orthorhombic test crystals: one or two atoms on a lattice whose three axes
differ, so that the mesh may have another number of points along each."""
import os

import numpy as np


def make_ortho(workdir, atoms, mesh, reach=1.3, **run):
    """Write the input files of the crystal with `atoms` (1: 3 bands, 2: 6 bands) atoms in the cell, Lennard-Jones
    pairs up to `reach` of the longest axis, and return their directory."""
    from ald import inputs as I
    abc, a = (1.0, 1.1, 1.23), 3.7 if atoms == 1 else 4.2
    red = [(0.0, 0.0, 0.0), (0.46, 0.5, 0.52)][:atoms]
    lj = I.lennard_jones(0.0104, 3.3)
    st = I.Structure(name="ortho-%d" % atoms, conv_abc=abc, prim_in_conv=np.eye(3), lattice_parameter=a,
                     atom_types=list(range(1, atoms + 1)), atom_red_conv=red, type_masses=[39.948, 83.798][:atoms],
                     type_names=["Ar", "Kr"][:atoms],
                     pairs=[(i, j, 0.1, reach * abc[2] * a, lj) for i in range(1, atoms + 1) for j in range(i, atoms + 1)])
    rp = I.RunParams(mesh=tuple(mesh))
    for k, v in run.items():
        setattr(rp, k, v)
    tag = "_".join(str(x) for x in mesh) + "".join("_%s%s" % kv for kv in sorted(run.items()))
    d = os.path.join(str(workdir), "ortho%d_%s_%s" % (atoms, reach, tag))
    if not os.path.exists(os.path.join(d, "fc3.dat")):
        I.write_inputs(st, rp, d)
    return d
