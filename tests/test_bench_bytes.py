"""The bytes that bench.py's fractions are of: what each path's launches read and write."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def test_a_step_is_measured_on_the_bytes_its_launches_move():
    import bench
    N, fc, elem = 1000, 100, 4
    for poynting in (True, False):
        launch, step = bench.algorithmic_bytes(N, fc, elem, poynting)
        # E, H and dt/eps read, E and H (and S) written; four auxiliary values a face cell, read and written
        assert step["ahead"] == step["fused"] == launch["k_tile_h (E ahead)"] == N * (18 if poynting else 15) * elem + fc * 8 * elem
        assert step["hs"] == launch["k_bulk_e"] + launch["k_tile_h"] == N * (24 if poynting else 21) * elem + fc * 8 * elem
        assert step["dropin"] == step["slab"] == sum(launch[k] for k in ("k_bulk_e", "k_bulk_h", "k_bulk_s"))
        assert step["dropin"] == N * (36 if poynting else 21) * elem + fc * 8 * elem
