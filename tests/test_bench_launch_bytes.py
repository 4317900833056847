"""The roofline bytes of the persistent inner launches (no GPU): the phases of
cgxx_b200/csrc/persist.cuh and the vectors it keeps in shared memory."""
import pytest

import bench

# (reads, writes) per phase; U is 16 bytes a row, G 8, vectors 4.
PHASES = {
    (2, True): [("U p", "q"), ("r q", "r"), ("G r", "y"), ("G y r C", "z"), ("p d z", "p d")],
    (2, False): [("U p", "q"), ("r q C", "r"), ("p r C d", "p d")],
    (1, True): [("U z p d", "d p q"), ("r q G", "r y"), ("G y r C", "z")],
    (1, False): [("U z p d", "d p q"), ("r q C", "r z")],
}
# In the iteration that stops: the split forms without y, z and the new p, then
# d += a p; the fused ones in full, then d += a p.
LAST = {
    (2, True): [("U p", "q"), ("r q", "r"), ("p d", "d")],
    (2, False): [("U p", "q"), ("r q C", "r"), ("p d", "d")],
    (1, True): PHASES[(1, True)] + [("p d", "d")],
    (1, False): PHASES[(1, False)] + [("p d", "d")],
}
# Accesses to a vector's resident copy. The split learned form's r: only the reads by
# its own rows, in the residual phase and beside z (it is always stored as well).
RESIDENT = {(2, True): {"z": 2, "d": 2, "q": 2, "r": 2}, (2, False): {"r": 3, "d": 2, "q": 2, "C": 2},
            (1, True): {"d": 2, "C": 1}, (1, False): {"r": 2, "d": 2, "q": 2, "C": 1}}


def size(names):
    return sum({"U": 16, "G": 8}.get(n, 4) for n in names.split())


@pytest.mark.parametrize("key", PHASES)
def test_launch_bytes_restate_the_phases(key):
    for phases, want in ((PHASES[key], bench.LAUNCH_BYTES[key][0]),
                         (LAST[key], bench.LAUNCH_BYTES[key][1])):
        assert sum(size(r) + size(w) for r, w in phases) == want
    assert {v: b // 4 for v, b in bench.LAUNCH_RESIDENT[key]} == RESIDENT[key]


def test_resident_vectors_fill_the_shared_memory_in_order():
    tile = bench.TILE_ROWS
    # One tile of each vector: all four fit.
    assert bench.resident_bytes((2, True), tile) == 32
    # 28 tiles (160^3): z whole, 20 tiles of d, no room for q and r.
    assert bench.resident_bytes((2, True), 160 ** 3) == pytest.approx(
        8 + 8 * 20 * tile / 160 ** 3)
    # More than 48 tiles: the first 48 of z.
    assert bench.resident_bytes((2, True), 96 * tile) == pytest.approx(8 * 48 / 96)


def test_launch_roofline_replaces_the_bytes():
    N = 160 ** 3
    results = [{"inner_form": 2}]
    roof = {"iterations_per_launch": 100.0, "launch_us": 7000.0, "peak": 6500.0,
            "algorithmic_bytes": 1.0, "achieved": 2.0, "frac": 3.0}
    out = bench.launch_roofline(roof, results, N, True)
    full = 96 - bench.resident_bytes((2, True), N)
    want = (99 * full + 48 - bench.resident_bytes((2, True), N)) * N
    assert out["algorithmic_bytes"] == pytest.approx(want)
    assert out["achieved"] == pytest.approx(want / 7e-3 / 1e9)
    assert out["frac"] == pytest.approx(out["achieved"] / 6500.0)
    assert out["all_in_memory_bytes"] == 1.0
