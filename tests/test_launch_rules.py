"""Host-side rules of the library's launches, seen through a recording stand-in for the CUDA runtime (CPU
only: no kernel runs)."""
import pytest
from launch_recorder import record

GRID = "(8, 4, 12, 16, 16)"   # nx, ny, nz, and the pitches of its layout


@pytest.mark.parametrize("call", [
    "L.lpb_apply_explicit_sym_f32(P(), P(), P(), P(), P(), *g, None)",
    "L.lpb_apply_explicit_sym_f64(P(), P(), P(), P(), P(), *g, None)",
    "L.lpb_apply_explicit_sym_noalloc_f32(P(), P(), P(), P(), *g, None)",
    "L.lpb_apply_explicit_modal_f32(P(), P(), P(), P(), P(), P(), P(), P(), *g, None)",
    "L.lpb_apply_explicit_modal_cheb_f32(2, None, P(), P(), P(), P(), P(), P(), P(), P(), P(), P(), P(), P(), *g, None)",
])
def test_explicit_apply_keeps_stream_order(tmp_path, call):
    """The cell pass of an explicit apply loads its matrices before it waits for the launch ahead, which may
    be the caller's own that writes them: the entries that promise stream order launch it in that order."""
    got = record(tmp_path, f"g = {GRID}\n{call}\nout = recorded()")
    cells = [r for r in got if r["what"] == "launch" and "_cells" in r["kernel"]]
    assert len(cells) == 1 and cells[0]["overlap"] == 0


@pytest.mark.parametrize("call", [
    "L.lpb_pack_sym_f32(P(), P(), 64, None)", "L.lpb_pack_sym_f64(P(), P(), 64, None)",
    "L.lpb_pack_modal_f32(P(), P(), P(), P(), P(), 64, 1e-6, None)",
    "L.lpb_chain_factor(P(), P(), P(), 16, 4, 4, 8, 8, None)",
])
def test_producers_of_early_loads_end_settled(tmp_path, call):
    """What an overlapping launch loads before its wait comes from passes that end with an empty launch,
    whose wait completes them."""
    got = [r for r in record(tmp_path, f"{call}\nout = recorded()") if r["what"] == "launch"]
    assert "settled" in got[-1]["kernel"] and len(got) > 1


def _limits_hold(records):
    """No limit is lowered, and every launch is within its kernel's limit from then on."""
    limit = {}
    for r in records:
        key = r["kernel"], r["device"]
        if r["what"] == "limit":
            assert r["bytes"] >= limit.get(key, 0), r
            limit[key] = r["bytes"]
        elif r["bytes"] > 48 * 1024:
            assert r["bytes"] <= limit.get(key, 0), r


@pytest.mark.parametrize("call", [
    "L.lpb_chain_solve_f32(P(), P(), P(), *grid(n), None)", "L.lpb_chain_solve_f64(P(), P(), P(), *grid(n), None)",
    "L.lpb_chain_solve_cols_f32(P(), P(), 1 << 20, 4, P(), *grid(n), None)",
    "L.lpb_band_inverse(P(), P(), P(), P(), *grid(n), None)",
])
def test_shared_memory_limits_are_never_lowered(tmp_path, call):
    """A kernel's dynamic shared-memory limit belongs to the process: a solve of a small level must not take it
    from under the launch of a large one that another thread is making."""
    body = f"""
def grid(n):
    p = (n[2] + 1 + 3) // 4 * 4
    return (*n, p, p)
for n in ((40, 10, 8), (6, 2, 2), (30, 10, 6), (40, 10, 8), (8, 3, 3)):
    assert {call} == 0
out = recorded()
"""
    _limits_hold(record(tmp_path, body))


@pytest.mark.parametrize("call", [
    *(f"L.lpb_apply_fine_{t}(P(), P(), P(), P(), host, P(), *g, None)" for t in ("f32", "f64")),
    *(f"L.lpb_apply_level1_{t}({m}, {f}, P(), P(), P(), None, None, None, P(), host, host, P(), *g, None)"
      for t in ("f32", "f64") for m, f in ((0, "P(), None, None, None, P(), None"), (1, "P(), P(), None, d, d, P()"),
                                           (2, "P(), d, P(), P(), d, P()"), (3, "P(), P(), P(), d, d, None"))),
])
def test_every_device_gets_its_limit(tmp_path, call):
    """The marches' shared-memory limits are set on each device that they run on."""
    body = f"""
from loadpath_b200.fem import hex8_ke
ke, modal = np.ascontiguousarray(hex8_ke(0.3, "im")), np.zeros(1024)
L.lpb_modal_ke(ke.ctypes.data, modal.ctypes.data)
g, d, host = (8, 4, 11, 12, 12), P(), modal.ctypes.data
for device in (0, 1, 0):
    on_device(device)
    assert {call} == 0
out = recorded()
"""
    got = record(tmp_path, body)
    assert {r["device"] for r in got if r["what"] == "launch"} == {0, 1}
    _limits_hold(got)


@pytest.mark.parametrize("reach,off", [(1, 0), (3, 0), (4, 0), (9, 0), (1, 8), (2, 8)])
def test_filters_past_the_march_go_tap_by_tap(tmp_path, reach, off):
    """Cones that reach further than the march stages, fields off the 16-byte boundary and all lists of the
    general entry take the many small blocks of the tap kernel."""
    args = f"P(), P() + {off}, P(), P(), 7, {{}}None, None, None, 3.0, 1e-9, 40, 20, 10, 12, 12, None"
    body = f"""
assert L.lpb_filter_reach({args.format(f"{reach}, ")}) == 0
a = recorded()
assert L.lpb_filter({args.format("")}) == 0
out = [[r["kernel"] for r in x if r["what"] == "launch"] for x in (a, recorded())]
"""
    named, general = record(tmp_path, body)
    assert len(named) == len(general) == 1 and "k_filter_taps" in general[0]
    assert ("k_filter_taps" if reach > 3 or off else "k_filter_march") in named[0]


@pytest.mark.parametrize("box,kernel", [
    ("0, 0, 0, 129, 65, 2", "k_patch_quads"),      # a z face: 128 patch cells in a tile's chunk
    ("0, 0, 0, 129, 65, 65", "k_patch_nodes"),     # supports on opposite faces
    ("0, 0, 0, 2, 65, 65", None),                  # an x face: 32, in the march
    ("0, 0, 0, 129, 2, 65", None),                 # a y face: 64
])
@pytest.mark.parametrize("mode", [0, 2])
def test_crowded_patch_cells_leave_the_march(tmp_path, box, kernel, mode):
    """On a grid of several units a block, patch cells stay in the level-1 march unless a tile's chunk may hold
    more of them than the block takes together."""
    fields = "P(), None, None, None, P(), None" if mode == 0 else "P(), d, P(), P(), d, P()"
    body = f"""
d, host, box = P(), np.ones(279), np.array([{box}], np.int32)
assert L.lpb_apply_level1_f32({mode}, {fields}, P(), P(), P(), P(), P(), P(), P(), host.ctypes.data, box.ctypes.data, P(),
                              128, 64, 64, 68, 68, None) == 0
out = [r["kernel"] for r in recorded() if r["what"] == "launch"]
"""
    got = record(tmp_path, body)
    assert "k_level1" in got[0] and len(got) == (1 if kernel is None else 2)
    assert kernel is None or kernel in got[1]


@pytest.mark.parametrize("fields", ["P() + 8, P()", "P(), P() + 8", "d, d"])
def test_level1_apply_refuses_what_it_cannot_address(tmp_path, fields):
    """An output or input off the 16-byte boundary, or the two the same, is refused before anything is launched."""
    body = f"""
from loadpath_b200._lib import LpError
d, host = P(), np.ones(279)
out = []
for fn in (L.lpb_apply_weights_tma_f32, L.lpb_apply_weights_tma_f64):
    try:
        fn({fields}, P(), None, None, P(), host.ctypes.data, None, P(), 8, 4, 11, 12, 12, None)
        out.append("taken")
    except LpError:
        out.append("refused")
out.append(sum(r["what"] == "launch" for r in recorded()))
"""
    assert record(tmp_path, body) == ["refused", "refused", 0]
