"""Downloads land in host memory whatever torch's default device is."""
import numpy as np
import torch


def test_download_with_another_default_device():
    from stonewall.fields import _download
    small, large = torch.arange(12.0).reshape(3, 4), torch.arange(1 << 20, dtype=torch.float64)
    with torch.device("meta"):
        a, b = _download(small), _download(large)
    np.testing.assert_array_equal(a, np.arange(12.0, dtype=np.float32).reshape(3, 4))
    np.testing.assert_array_equal(b, np.arange(1 << 20))
