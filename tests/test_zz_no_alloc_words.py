"""epi_tick_hour_noalloc on house and office words that name no cell of the plane: the call says so
(EPI_ERR_INVARIANT), moves nobody out of the plane and leaves the plane's border alone; a sound
world runs as before right after it.

The words' halves lie at and beyond the ends of what packed cells can be compared in (14 and 15
bits, and ones whose borrow reaches the other half)."""
import ctypes as C
import json

import numpy as np
import pytest

from helpers import COVID_FAST, make_config
from test_zz_no_alloc import _pack

pytestmark = pytest.mark.gpu

EPI_ERR_INVARIANT = 5
WORDS = [0xFFFFFFFF, 0xFFFF0000, 0x0000FFFF, 0x80008000, 0x40004000, 0x7FFF7FFF, 0x3FFF3FFF, 0xBFFFBFFF]


@pytest.mark.parametrize("hour", [24 * 7 + 7, 24 * 7 + 8, 24 * 7 + 9, 24 * 7 + 12, 24 * 7 + 16, 24 * 7 + 23])
def test_words_outside_the_plane_are_reported(gpu, hour):
    import torch

    from epirust_gb300 import Config, Epidemiology, lib
    from epirust_gb300._lib import EpiGeography

    config = Config(json.dumps(make_config(n=4000, grid=120, seed=21, disease=COVID_FAST, starting=(5, 5, 5, 30))))
    p, L = config.params, lib()
    G = p.grid_size
    geo = EpiGeography()
    assert L.epi_define_geography(G, C.byref(geo)) == 0
    assert L.epi_resize_hospital(C.byref(geo), p.number_of_agents, 0.002, p.hospital_beds_percentage) == 0
    base = Epidemiology(config)
    base.simulate_hours(1, hour - 1)
    world = base.snapshot()
    base.close()
    sound = _pack(world, p, geo, (geo.hospital.x0, geo.hospital.y0, G, G))

    def call(arrays):
        t = [torch.from_numpy(a.copy().view(np.int32) if a.dtype == np.uint32 else a.copy()).cuda() for a in arrays]
        counts = torch.zeros(8, dtype=torch.int32, device="cuda")
        rc = L.epi_tick_hour_noalloc(C.byref(p), hour, 0, *[a.data_ptr() for a in t], counts.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
        return rc, [a.cpu().numpy() for a in t], counts.cpu().numpy()

    rc, want, want_counts = call(sound)
    assert rc == 0
    for word in WORDS:
        pos, state, home, work, wsa, plane = [a.copy() for a in sound]
        home[::2] = word
        work[::3] = word
        state[::40] &= ~np.uint32(7)  # at hour 23 some of them walk home recovered
        state[::40] |= np.uint32(6 if hour % 24 == 23 else 0)
        rc, out, _ = call([pos, state, home, work, wsa, plane])
        assert rc == EPI_ERR_INVARIANT, hex(word)
        moved = out[0].view(np.uint32)
        assert (moved & 0xFFFF).max() <= G and (moved >> 16).max() <= G, hex(word)
        cells = out[5][: (G + 3) * (G + 3)].reshape(G + 3, G + 3)
        assert not (cells[0].any() or cells[-1].any() or cells[:, 0].any() or cells[:, -1].any())
        assert int((out[5] != 0).sum()) == len(world)
    rc, again, again_counts = call(sound)
    assert rc == 0 and (again_counts == want_counts).all()
    assert all((a == b).all() for a, b in zip(again, want))
