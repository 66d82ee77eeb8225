"""The executor's tests once more with everything through the ranks' slots, as between GPUs: a launch that carries all ranks on one GPU otherwise runs the call's data flow."""
import pytest

from test_executor_gpu import *      # noqa: F401,F403
from test_executor_gpu import pytestmark      # noqa: F401


@pytest.fixture(autouse=True, scope="module")
def through_the_slots():
    from piccl_b200.parallel import comm

    class SlotsOnly(comm.LoopbackGroup):
        def __init__(self, *a, **kw):
            super().__init__(*a, **kw)
            self.slots_only()
    with pytest.MonkeyPatch.context() as m:
        m.setattr(comm, "LoopbackGroup", SlotsOnly)
        yield


del test_data_flow_is_the_programs_bit_for_bit, test_slices_of_a_data_flow      # noqa: F821
