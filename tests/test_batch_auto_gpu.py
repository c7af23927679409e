"""GPU: GL_BATCH_AUTO takes the mode tuned for the batch's shape, seen in the
launches that are recorded (those inside a graph or the persistent kernel are not)."""
import json

import pytest

from conftest import rand_field, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["persistent", "buckets", "per_call"])
def test_tuned_mode_is_taken(gl, cuda, tmp_path, mode):
    from goldilocks_gb300 import _lib as L, batch, tune
    lens, dirs = [512, 1024, 1024], [0, 1, 0]
    f = tmp_path / "t.json"
    f.write_text(json.dumps({"format": "goldilocks-gb300-tuning", "version": 1,
                             "batches": [{"mode": mode, "polys": list(map(list, zip(lens, dirs)))}]}))
    x = to_dev(cuda, rand_field(2560, seed=1))
    want = x.clone()
    for at, n, d in zip([0, 512, 1536], lens, dirs):
        (gl.intt if d else gl.ntt)(want[at:at + n])
    lib = L.load()
    tune.load(str(f))
    try:
        lib.gl_profile_enable(1)
        batch.run_packed(x, [0, 512, 1536], lens, dirs)
        recorded = lib.gl_profile_read(None, 0)
    finally:
        lib.gl_profile_enable(0)
        tune.clear()
    assert cuda.equal(x, want)
    assert (recorded > 0) == (mode == "per_call")
