"""The autotuner's cache across builds: an FP64 line timed with passes in FP64 arithmetic is
not applied to the fixed-point passes, other lines still are."""
import json

import pytest

from _helpers import configs

pytestmark = pytest.mark.gpu
N = (32, 32, 32)
OTHER = dict(y_tx=4, z_tx=4, x_fused=1, y_pairs=0, fuse_stage=0, z_split=2, y_prefetch=0, overlap=0, slab_pipe=0,
             zf_pipe=1)


def tuned(precision, cache):
    import gturbo3d_gb300 as g
    gp, _ = configs(N, precision=precision, forcing="none")
    with g.Simulation(gp) as sim:
        ms = g.api.autotune(sim, str(cache))
        return ms, {k: sim.get_tuning(k) for k in OTHER}


def line(key):
    return json.dumps({"key": key, **OTHER, "ms_per_step": 0.001}) + "\n"


def test_fp64_line_of_other_passes_is_ignored(lib, tmp_path):
    torch = pytest.importorskip("torch")
    name = torch.cuda.get_device_name(0).replace(" ", "_")
    cache = tmp_path / "old.jsonl"
    cache.write_text(line(f"32x32x32/fp64/pruned/{name}"))
    ms, knobs = tuned("fp64", cache)
    assert ms > 0                                           # timed, not taken from the line
    assert knobs["y_tx"] == 0 and knobs["z_tx"] == 0        # no effect on these passes: not searched
    assert tuned("fp64", cache) == (-1.0, knobs)            # its own line


def test_mixed_line_is_still_taken(lib, tmp_path):
    torch = pytest.importorskip("torch")
    name = torch.cuda.get_device_name(0).replace(" ", "_")
    cache = tmp_path / "old.jsonl"
    cache.write_text(line(f"32x32x32/mixed/pruned/{name}"))
    assert tuned("mixed", cache) == (-1.0, OTHER)
