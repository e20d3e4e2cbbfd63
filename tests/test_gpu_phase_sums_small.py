"""Far-field sums of few particles, on both sides of the rule that chooses their kernel; checks and bounds of
test_gpu_phase_sums.py."""
import pytest

from test_gpu_phase_sums import test_far_field_sum as _far_field_sum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 11])
@pytest.mark.parametrize("R,m_max", [(1, 0), (2, 3), (3, 1), (4, 4), (16, 3), (16, 4), (5, 2)])
def test_few_particles(n, R, m_max, gpu_context):
    _far_field_sum(n, R, m_max, 3, 130, 1e4, gpu_context)
