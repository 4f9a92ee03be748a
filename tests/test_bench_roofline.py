"""bench.py's roofline entry on made-up profiles: the kernel it names is the
one that the timed steps launch."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402

INFO = {"nodes": 1000, "matvec_bytes_fp64": 480e3, "matvec_bytes_fp32": 272e3, "columns": 100, "elements": 900}


class _Problem:
    """Stands for a problem whose runs take the resident PCG (or not)."""

    def __init__(self, resident):
        self.is_resident, self.preps, self.mode = resident, [], None
        self.preps = [type("P", (), {"inputs": type("I", (), {"guess_mode": 1, "precision": 0})})()]

    def timing(self, enable, as_run=False):
        if enable:
            self.mode = as_run

    def set_guess(self, u, v):
        pass

    def run(self):
        return [{"pcg_iters_total": 40}]

    def resident(self):
        return self.is_resident

    def kernel_times(self):
        assert self.mode is True  # the kernels of the timed steps
        mv = (0.2, 2) if self.is_resident else (0.4, 40)
        upd = (0.0, 0) if self.is_resident else (0.3, 80)
        return {"pcg_matvec_fp64": mv, "pcg_update_fp64": upd, "assembly_qp": (0.1, 2), "assembly_rows": (0.1, 2)}

    def mv_nodes(self):
        return (0.0 if self.is_resident else 40e3), 0.0, 0, 0

    def info(self):
        return dict(INFO)


def _roof(*resident):
    kp = bench.kernel_profile({"probs": [_Problem(r) for r in resident]}, None)
    return kp, bench.roofline(kp, "standard", False, 6483.9, "measured", None)


def test_roofline_names_the_kernel_of_the_timed_path():
    kp, r = _roof(True)
    assert "k_pcg_resident" in r["kernel"] and r["bound"] == "latency" and r["launches_timed"] == 2
    assert abs(r["us_per_iteration"] - 5.0) < 1e-9 and kp["launches"] == 6
    assert abs(r["achieved"] - 2 * 480e3 / 0.2e-3 / 1e9) < 0.1
    kp, r = _roof(False)
    assert "k_std_mv" in r["kernel"] and r["bound"] == "hbm" and r["launches_timed"] == 40
    assert abs(r["achieved"] - 40 * 480e3 / 0.4e-3 / 1e9) < 0.1 and kp["launches"] == 124
    _, r = _roof(True, False, True)  # 0.4 ms resident, 0.4 ms launched: the matvec
    assert "k_std_mv" in r["kernel"]
    _, r = _roof(True, False, True, True)
    assert "k_pcg_resident" in r["kernel"]
