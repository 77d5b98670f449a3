"""A tune-cache file outlives the face kernels that its layouts were timed with."""
from __future__ import annotations

import json

import pytest

import umcp_gb300 as U
from conftest import load_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [U.FP64, U.FP32_CENTRED])
def test_layouts_of_other_kernels_are_timed_anew(tmp_path, precision):
    """An entry without the kernels' version, as files from before it hold them, is neither used nor lost."""
    cache = tmp_path / "tune.json"
    ctx = U.Context(0)

    def run():
        batch = U.Batch(ctx, precision, tune_cache=cache)
        plan, prm, _ = load_case("ico3_deformed", precision)
        mesh = U.Mesh(ctx, plan, prm)
        batch.add(mesh, U.integrator(U.OVERDAMPED_BD, time_step=1.0, D=1e-4, seed=3), 0, 8)
        batch.run(8)
        return batch.info(), mesh

    first, _ = run()
    (key, choice), = json.loads(cache.read_text()).items()
    old_key = "|".join(key.split("|")[:4])  # device, precision, patch types, log2 of faces
    old = dict(choice, tile_faces=choice["tile_faces"] * 2, blocks_per_sm=1, face_ms=99.0)
    # the file's own layout: an entry a line
    cache.write_text('{\n  "%s": %s\n}\n' % (old_key, json.dumps(old)))
    second, _ = run()
    assert first.tune_source == second.tune_source == 1 and second.tuned_face_ms != 99.0
    entries = json.loads(cache.read_text())
    assert entries[old_key] == old and set(entries) == {old_key, key}
    third, _ = run()
    assert third.tune_source == 2 and third.tuned_face_ms == pytest.approx(entries[key]["face_ms"], abs=1e-6)
