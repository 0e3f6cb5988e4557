"""One context per host thread, each with a stream and a subset size of its own:
frames of different shared-memory sizes launched side by side.  The limit of a
kernel's dynamic shared memory belongs to the process, so that a thread that
lowers it between another's setting and launch makes that launch fail."""
import threading

import numpy as np
import pytest

from dice_b200 import abi
from dice_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subsets,step", [((11, 21, 31, 37), 40), ((41, 51, 61, 71), 9)])   # rows; lean, and rows beside it
def test_contexts_in_threads(subsets, step):
    torch = pytest.importorskip("torch")
    from dice_b200.schema import Schema
    size, frames = (200, 300) if step == 40 else (640, 40)
    ref = syn.speckle_image(size, size, seed=1, blur_sigma=0.8).numpy()
    deff = syn.warp_image(torch.from_numpy(ref), lambda X, Y: (0.3 + 0 * X, -0.2 + 0 * Y), noise_sigma=1.0, seed=2).numpy()
    out, errors = {}, []
    start = threading.Barrier(len(subsets))

    def run(subset, key, n, wait):
        try:
            cx, cy = syn.grid_points(size, size, subset, step)
            p = abi.default_params(subset_size=subset, enable_rotation=1, enable_normal_strain=1, enable_shear_strain=1,
                                   fast_solver_tolerance=1e-3, optimization=abi.GRADIENT_BASED)
            with Schema(p, stream=torch.cuda.Stream()) as s:
                s.set_ref_image(ref)
                s.set_fields(syn.init_fields(cx, cy))
                s.set_def_image(deff)
                rows = torch.from_numpy(syn.init_fields(cx, cy)).cuda()
                torch.cuda.synchronize()
                if wait:
                    start.wait()
                for _ in range(n):
                    s.load_fields(rows)
                    s.execute_correlation()
                out[key] = s.fields()
        except Exception as e:   # noqa: BLE001 (reported by the main thread)
            errors.append((subset, e))
            start.abort()

    for subset in subsets:
        run(subset, (subset, "alone"), 1, False)
    assert not errors, errors
    threads = [threading.Thread(target=run, args=(s, (s, "beside"), frames, True)) for s in subsets]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s in subsets:
        assert np.array_equal(out[(s, "alone")], out[(s, "beside")])
