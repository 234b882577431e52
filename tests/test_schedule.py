"""The step's default schedule (schedule.default_mode)."""

import pytest

from newton_custom_contact_b200.schedule import default_mode


@pytest.mark.parametrize("bodies,want", [(1, ("groups", 32)), (62, ("groups", 32)), (63, ("groups_compact", 32)),
                                         (128, ("groups_compact", 32)), (129, ("groups_compact", 64)),
                                         (512, ("groups_compact", 128)), (513, ("batch", None))])
def test_default_mode_without_a_world_count(bodies, want):
    # by the largest world alone: the smallest group that holds it
    assert default_mode(bodies) == want
