"""The tensor X-engine's load ring, checked on the CPU through corrx_tc_geometry: two
converter groups take alternate stages, and a slot's loads must all be one group's, or
its wait on the slot's phase parity could take an earlier load for the one it wants."""

from __future__ import annotations

import ctypes as C

import pytest

GROUPS = 2


@pytest.mark.parametrize("split", [False, True])
def test_a_slot_belongs_to_one_group(pkg, split):
    lib = pkg.abi.load()
    shapes = 0
    for n in range(1, 65):
        for ct in (2, 4, 8):
            for kt in (16, 32, 64):
                g = pkg.abi.corrx_tc_geom(struct_size=C.sizeof(pkg.abi.corrx_tc_geom))
                pkg.abi.check(lib.corrx_tc_geometry(n, int(split), ct, kt, C.byref(g)),
                              "corrx_tc_geometry")
                if not g.ok:
                    continue
                shapes += 1
                assert g.n_ld >= GROUPS and g.n_ld % GROUPS == 0, (n, ct, kt, g.n_ld)
    assert shapes > 100
