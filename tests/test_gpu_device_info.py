"""The device a context reports is the one it runs on."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_device_name():
    import prt
    c = prt.Context(0)
    assert c.info() == torch.cuda.get_device_name(0)
    c.close()
