"""The mesh's edge parameter compares a float with 1e-6 in double in the
reference; the kernels compare with the float 1e-6f.  The same for every float:
1e-6f is the largest float below 1e-6."""
import numpy as np


def test_threshold():
    f = np.float32(1e-6)
    assert float(f) < 1e-6 < float(np.nextafter(f, np.float32(1)))
    x = np.concatenate([np.arange(-4000, 4000, dtype=np.int32) + f.view(np.int32),
                        np.linspace(0, 0x7f800000, 100001).astype(np.int32)]).view(np.float32)
    assert np.array_equal(x.astype(np.float64) < 1e-6, x <= f)
