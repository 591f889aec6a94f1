"""The autotuner's candidates and cache keys, on the host."""
import json
from types import SimpleNamespace

import pytest

from dtmm_gb300.tune import Autotuner, col_tiles, schedules, tuning_key


def _plan(height, width, precision, method=4, real_path=1):
    d = SimpleNamespace(height=height, width=width, method=method, diffraction=3, npol=2, nray=1, real_path=real_path)
    return SimpleNamespace(desc=d, precision=precision)


@pytest.mark.parametrize("shape", [(256, 256), (150, 210), (250, 330), (64, 64), (45, 1024)])
@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_two_step_transforms_are_timed(shape, precision):
    """Both precisions transform these sides in registers by default: a tuned plan may keep doing so."""
    s = schedules(_plan(*shape, precision))
    assert s[0] == 1 and 2 in s and (3 in s) == (shape[0] % 8 == 0 or shape[1] % 8 == 0)


def test_column_tiles_are_different_launches():
    # 16 lines a block: 16 // 4 columns of four components, 16 // 2 of two
    assert max(col_tiles(_plan(256, 256, "mixed"), 1)) == 4
    assert max(col_tiles(_plan(256, 256, "mixed", method=2), 1)) == 8
    assert max(col_tiles(_plan(256, 256, "mixed"), 2)) == 16


def test_picks_of_earlier_passes_lapse(tmp_path):
    """Keys as they were before the line kernels are not found again; new ones are."""
    plan = _plan(256, 256, "double")
    old = {"256x256/m4/double/d3/f2": dict(fft_schedule=3, row_group=2, col_tile=8)}
    path = tmp_path / "tuned.json"
    path.write_text(json.dumps(old))
    t = Autotuner(path=str(path))
    assert t.lookup(plan) is None
    t.cache[tuning_key(plan)] = dict(fft_schedule=1, row_group=0, col_tile=0)
    t.save()
    assert Autotuner(path=str(path)).lookup(plan) == dict(fft_schedule=1, row_group=0, col_tile=0)


def test_complex_records_have_their_own_picks():
    assert tuning_key(_plan(64, 64, "mixed")) != tuning_key(_plan(64, 64, "mixed", real_path=0))
