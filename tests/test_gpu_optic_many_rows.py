"""The optic substep's shapes on both sides of the row count above which rows take half a warp."""
import pytest

from test_gpu_optic_shapes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [47_360, 47_361])
@pytest.mark.parametrize("batch", [3, 5, 6, 7, 8, 12, 20])
def test_lobes_around_the_line_of_many_rows_match_oracle(m, batch):
    check(m, batch)


@pytest.mark.parametrize("launch", ["persistent", "step"])
def test_three_flies_in_lobes_of_few_and_more_rows(launch):
    for m in (9472, 9473):
        check(m, 3, launch=launch)
