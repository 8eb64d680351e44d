"""Substeps at the sizes where the line solves, the right-hand side's row blocks
and the packed x transforms change form, against the numpy restatement:

* k_line's chunks of 16 rows: one short chunk, exactly full ones, a last chunk
  of one row (where w, one row shorter, has none), the tallest partitioned
  column (192 rows) and the first whole-column one (193);
* planes whose columns do not fill the last group of 16 (or of 32), odd and even;
* whole columns of even planes at both orders, by their height (193 rows, several
  partial tiles) and by their plane (more than 111 tiles), fewer rows than the back
  sweep reads ahead;
* rows that k_rhs's blocks do not divide: last blocks of one row and of two, in both
  schemes;
* x transforms of two columns each: an odd last column, 16-column blocks with
  one column and with fifteen;
* transforms planned at run time: one stage (4, 5), the largest size (500),
  each radix first and last, lines that do not fill a block of 8;
* the divergence's loads ahead: a plane's last positions that fill part of a
  turn of 16, with fixed (48, 192, 320) and planned sizes.

Bars as test_gpu_parity.py: relative L2 1e-13 on u, v, w, c and 1e-10 on p
(rounding of u* by 1e-16 is divided by dt and passes the inverse Laplacian),
1e-9 of the column scale on the log, and for the two control values at least
1e-14 / dt."""
import numpy as np
import pytest

import chanfast_np as cn
import ic
from perf import cases

pytestmark = pytest.mark.gpu

CASES = [(2, 12, 15, 4), (4, 10, 9, 6), (2, 16, 18, 15), (4, 15, 81, 16), (2, 9, 16, 17), (4, 8, 25, 17),
         (4, 12, 30, 32), (2, 15, 45, 33), (4, 20, 6, 49), (4, 6, 5, 192), (2, 6, 5, 193), (4, 8, 10, 193)]
TRANSFORMS = [(2, 500, 4, 4), (4, 5, 500, 6), (2, 4, 486, 5), (4, 243, 8, 6), (2, 40, 24, 4), (4, 200, 250, 6),
              (4, 48, 18, 7), (2, 192, 30, 5), (4, 192, 9, 6), (4, 320, 15, 6)]


WHOLE = [(2, 40, 72, 193), (4, 40, 72, 193), (2, 200, 160, 9), (4, 200, 160, 9), (2, 200, 160, 4)]
# on 148 SMs blocks of 7 rows and a last one of 1 (43) or 2 (37)
SHORT_BLOCKS = [(2, 64, 64, 43), (4, 64, 64, 43), (2, 64, 64, 37), (4, 64, 64, 37)]


@pytest.mark.parametrize("order,nx,ny,nz", CASES + TRANSFORMS + WHOLE + SHORT_BLOCKS)
def test_substeps_match_restatement(cf, gpu, order, nx, ny, nz):
    prm = cn.Params(order=order, nx=nx, ny=ny, nz=nz, lx=2 * np.pi, ly=np.pi, lz=2.0, dt=1e-3, nu=1.0 / 3000.0,
                    prandtl=0.71, setuframe=0.3, betg_x=0.1, betg_y=0.05, betg_z=0.02)
    g = cn.Grid(prm)
    u, v, w, c = ic.raw_state(prm, g.dz, 11, 0.1, 0.01)
    cn.project_initial(u, v, w, prm, g, 1.0)
    st = cn.new_state(u, v, w, c, g)
    with cf.Instance(cf.Config.from_params(prm)) as inst:
        for nm, a in zip("uvwc", (u, v, w, c)):
            inst.set_field(nm, a)
        inst.step(4)
        inst.sync()
        cn.run(st, prm, g, 4)
        I = (slice(3, 3 + nx), slice(3, 3 + ny), slice(3, 3 + nz))
        for nm in "uvwcp":
            a, b = inst.get_field(nm)[I], getattr(st, nm)[I]
            rel = np.linalg.norm(a - b) / np.linalg.norm(b)
            assert rel <= (1e-10 if nm == "p" else 1e-13), (nm, rel)
        log, ref = inst.log(), np.array(st.log)
        assert log.shape == ref.shape
        bar = 1e-9 * np.maximum(np.abs(ref).max(axis=0), 1e-3)
        bar[[0, 5]] = np.maximum(bar[[0, 5]], 1e-14 / prm.dt)
        assert np.all(np.abs(log - ref) <= bar), np.abs(log - ref).max(axis=0)


@pytest.mark.parametrize("order,nz", [(2, 43), (4, 43), (2, 37), (4, 37)])
def test_fully_implicit_scheme_with_short_blocks(cf, gpu, order, nz):
    """Its right-hand side takes the same row blocks: against the plain 64-bit
    torch statement of the scheme.  Bars as test_gpu_channel.py: 1e-12 on
    u, v, w, c and 1e-10 on p."""
    case = cases.flow("short", "step", order, 64, 64, nz, 1, scheme="channel", re=100.0, dt=1e-3, betg=0.1, uframe=0.3)
    state = cases.prepare(case, 5)
    got = cases.run(state)
    state["inst"].sync()
    want = cases.exact(case, 5)
    for nm in "uvwcp":
        rel = float((got[nm] - want[nm]).norm() / want[nm].norm())
        assert rel <= (1e-10 if nm == "p" else 1e-12), (nm, rel)
    state["inst"].close()


def test_batch_of_odd_and_even_planes_matches_plain(cf, gpu):
    """Odd and even planes, partitioned and whole columns, in launches of their
    own: against the plain path (test_gpu_batch.py: bit for bit)."""
    out = []
    for batched in (False, True):
        insts = []
        for q, (order, nx, ny, nz) in enumerate([(2, 12, 15, 10), (4, 10, 9, 12), (4, 12, 16, 20), (2, 48, 40, 33)]):
            inst = cf.Instance(cf.Config.make(order, nx, ny, nz, 2 * np.pi, np.pi, 2.0, 1e-3, 1.0 / 3000.0, prandtl=0.71,
                                              betg_y=0.05))
            inst.init_fields(q, 0.1, 0.01)
            insts.append(inst)
        if batched:
            cf.batch_step(insts, 6)
        else:
            for inst in insts:
                inst.step(6)
        for inst in insts:
            inst.sync()
        out.append([{nm: inst.get_field(nm, cf.LAYOUT_INTERIOR) for nm in "uvwcp"} for inst in insts])
        for inst in insts:
            inst.close()
    for a, b in zip(*out):
        for nm in "uvwcp":
            assert np.linalg.norm(a[nm] - b[nm]) <= (1e-10 if nm == "p" else 1e-13) * np.linalg.norm(a[nm]), nm
