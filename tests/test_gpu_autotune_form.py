"""skc_autotune searches the bitmap kernel's parameters (grid depth, tile, chunk,
CTAs per SM) only where the bitmap kernel runs: the other forms ignore them, and
what their noise prefers would be stored for datasets that take the bitmaps."""
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,opts", [
    ("skyline", {"subspace": 0b1011}),
    ("cuboids", {"algo": "sdsc", "mode": "plain", "max_d": 2}),
    ("levels", {"max_d": 2, "form": "levels"}),
    ("bitmaps", {"max_d": 2, "form": "bitmaps"})])
def test_parameters_of_other_forms_are_left_alone(gpu_ctx, form, opts):
    opts = dict(opts, pq_size=64)
    ds = sk.Dataset(gpu_ctx, datagen.generate("anticorrelated", 40000, 8, 11))
    try:
        r = sk.skycube(gpu_ctx, ds, **opts)  # also makes the dataset's signature
        assert r.form()[0] == form
        r.close()
        sk.signature(ds)
        a = sk.kernel_launches()
        sk.skycube(gpu_ctx, ds, **opts).close()
        b = sk.kernel_launches()
        params, _ = sk.autotune(gpu_ctx, ds, repeats=1, **opts)
        runs = (sk.kernel_launches() - b) / (b - a)
        if form == "bitmaps":
            assert runs > 6
        else:
            assert runs == 1
            assert (params["depth"], params["tile_points"], params["chunk"],
                    params["blocks_per_sm"]) == (7, 256, 1, 0)
    finally:
        gpu_ctx.tuning_clear()
    ds.close()
