"""One object per device, however it is asked for, and nothing but text and devices names one."""
import copy
import pickle

import pytest

from mytorch_b200.tensor import Device


@pytest.mark.parametrize("wrong", [None, 3, ("cuda", 0), [1], b"cuda"])
def test_only_text_and_devices_name_a_device(wrong):
    Device("cuda:0")
    with pytest.raises((AttributeError, TypeError)):
        Device(wrong)


def test_one_object_per_device():
    assert Device("cuda:0") is Device(" cuda : 0 ") is Device(device=Device("cuda:0")) is pickle.loads(pickle.dumps(Device("cuda:0")))
    assert copy.deepcopy(Device("cpu")) is Device("cpu") is not Device("cuda")
