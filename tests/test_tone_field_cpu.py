"""A tone field's device form from tones of any number, none included."""
import numpy as np
import pytest

import spinsim_b200 as ss


@pytest.mark.parametrize("tones,rate", [({}, 1), ({0: []}, 1), ({0: np.zeros((0, 3)), 2: [[3.5, 1.0, 0.0]]}, 4),
                                        ({1: [[-7e6, 2.0, 0.1], [2e3, 1.0, 0.0]]}, 7_000_000), ({0: [[1e300, 1.0, 0.0]]}, 10 ** 18), ({0: [[np.nan, 1.0, 0.0], [9.0, 1.0, 0.0]]}, 9)])
def test_device_struct(tones, rate):
    field = ss.ToneField(tones, bias=[0.0, 0.0, 5.0])
    f, keep = field.device_struct("cpu")
    assert f.n_params == rate
    assert [f.tone_count[c] for c in range(3)] == [len(tones.get(c, ())) for c in range(3)]
    assert f.bias[2] == 5.0 and all(t.device.type == "cpu" for t in keep)
