"""Calls at the far end of the sizes that the entry points take."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [2**31 - 1, 2**31 - 1024])
def test_boxcar_of_the_longest_series(vf, nt):
    """The last tile of the longest series (8.6 GB): a pulse in its last four samples
    is found where it is, with the SNR of four samples of 3 at sigma 1, 12 / 2, exactly."""
    import torch
    if torch.cuda.mem_get_info()[0] < 10 << 30:
        pytest.skip("needs 10 GB")
    x = torch.zeros((1, nt), device="cuda")
    x[0, nt - 4:] = 3.0
    snr, start, width = vf.boxcar(x, torch.zeros(1, device="cuda"), torch.ones(1, device="cuda"), 4)
    assert (float(snr), int(start), int(width)) == (6.0, nt - 4, 4)
