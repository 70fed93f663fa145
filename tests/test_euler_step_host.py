"""``Euler`` reads its time step and material at every step, in the pair form as
in the others (no GPU: the library's call is replaced)."""
import types

from probabilistic_peridynamics_gb300 import Euler, _lib, integrators


def test_numbers_are_read_at_every_step(monkeypatch):
    seen = []

    def step(args, pairs, stream):
        a = args._obj
        seen.append((a.dt, a.bond_stiffness, a.critical_strain, a.bc_scale,
                     a.force_bc_scale))
        return _lib.PP_SUCCESS

    e = Euler(dt=0.5)
    monkeypatch.setattr(integrators, "lib", lambda: types.SimpleNamespace(
        pp_cy_pair_step=step))
    e._device = types.SimpleNamespace(stream_handle=None)
    e.nnodes, e._width = 2, 1
    e.bond_stiffness, e.critical_stretch = 3.0, 0.1
    for name in ("coords", "volume", "fc_values", "fc_types", "bc_values",
                 "bc_types", "nlist", "n_neigh", "force", "u"):
        setattr(e, f"_{name}_d", None)
    e._step = e._make_step()
    e._pairs = types.SimpleNamespace(struct=_lib.CyPairs())
    e(0.01, 0.02)
    e.dt, e.bond_stiffness, e.critical_stretch = 0.25, 4.0, 0.2
    e(0.03, 0.04)
    assert seen == [(0.5, 3.0, 0.1, 0.01, 0.02), (0.25, 4.0, 0.2, 0.03, 0.04)]
