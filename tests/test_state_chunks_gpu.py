"""The state-space mixer where the state has more than 64 channels: the wide tiles of the chunks' sums, whole and ragged."""
import pytest

import test_rorutar_gpu as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads, vdim, state, groups, taps, parts", [(2, 64, 128, 1, 4, 1), (2, 40, 72, 2, 4, 1), (4, 10, 130, 2, 3, 2),
                                                                     (2, 72, 66, 1, 2, 1)])
def test_wide_states(dtype, heads, vdim, state, groups, taps, parts):
    R.test_state_space(dtype, heads, vdim, state, groups, taps, parts)
