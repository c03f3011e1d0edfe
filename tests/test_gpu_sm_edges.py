"""The sizes where a launch changes with the number of SMs, taken from the device: the edge tests
of training, inference, few spectra and the index build list them for 152 SMs."""
import pytest

import tests.test_gpu_build_edges as build
import tests.test_gpu_few_spectra as few
import tests.test_gpu_mlp_training as mlp

pytestmark = pytest.mark.gpu


def _sms() -> int:
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("rows", [8, 16, 32])
def test_training_tiles(rows):
    """8, 16 and 32 rows an SM: the tile grows past the first two, a CTA takes two past the last."""
    for n in (rows * _sms(), rows * _sms() + 1):
        mlp.test_gradients_at_tile_edges(n)


@pytest.mark.parametrize("rows,past", [(16, 1), (32, 1), (64, 1), (64, 33), (96, 1), (128, 1)])
def test_inference_tiles(rows, past):
    """16 spectra an SM: rows or tiles; half tiles up to 32 past whole waves of 64."""
    for n in (rows * _sms(), rows * _sms() + past):
        mlp.test_inference_at_tile_edges(n)


@pytest.mark.parametrize("share", [8, 4, 2])
def test_spectra_in_parts(share):
    """One spectrum in eight SMs: shorter parts; one in two: none."""
    for n in (_sms() // share, _sms() // share + 1):
        few.test_few_spectra_equal_oracle(n)


def test_sort_tiles():
    """16 postings an entry: up to a tile of 2048 of them for every SM, then tiles of 8192."""
    for npep in (128 * _sms() - 1, 128 * _sms(), 128 * _sms() + 1):
        build.test_entry_order_at_sort_edges(npep)
