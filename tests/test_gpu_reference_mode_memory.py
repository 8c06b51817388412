"""Reference mode on a device without room for the packed node records: the
engine walks over the tree's own arrays and gives the same forces, bit for bit
(the records hold the same values)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_no_room_for_the_records(precision, monkeypatch):
    from cnb.core import engine as engine_module
    from cnb.core.state import SimulationState
    from cnb.utils import config as cfgmod
    from cnb.utils.cosmology import zeldovich_arrays
    cfg = cfgmod.make(N_GRID=16, SOFTENING=0.5 / 16, THETA=0.6, N_STEPS=100, A_START=0.02, A_END=0.22,
                      KEY_MODE="morton63", FORCE_MODE="reference", PRECISION=precision)
    forces = []
    for full in (False, True):
        real = torch.empty

        def empty(*args, **kwargs):
            if full and args and args[0] == (4, 2 * 16 ** 3 - 1, 4):
                raise torch.cuda.OutOfMemoryError("no room")
            return real(*args, **kwargs)

        st = SimulationState(16 ** 3, *zeldovich_arrays(16, 1))
        with monkeypatch.context() as m:
            m.setattr(torch, "empty", empty)
            eng = engine_module.SimulationEngine(cfg, st, camera=False)
        assert (eng.ref_table is None) == full
        for _ in range(2):
            eng.step()
        eng.check()
        forces.append(st.force.clone())
    assert bool((forces[0].view(torch.int32) == forces[1].view(torch.int32)).all())
