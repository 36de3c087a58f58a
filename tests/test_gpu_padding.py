"""The scan padding without padded counts (qssb_pad_fill, qssb_pad_columns):
fill pattern, sums and columns bit for bit against a padded block made with
numpy, at odd scans and borders, and a session against one given the padded
block."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import ssb_oracle as so
from quantem.gpu_b200 import B200SSBBackend, _lib, ops
from quantem.gpu_b200.synthetic import CONFIGS, generate

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("scan", [(1, 1), (127, 128), (128, 3), (33, 95), (121, 64)])
@pytest.mark.parametrize("npix", [8, 13])
def test_fill_sums_and_columns_are_those_of_the_padded_block(scan, npix):
    rng = np.random.default_rng(scan[0] * 1000 + scan[1] + npix)
    data = rng.integers(0, 65536, (*scan, npix, 1), dtype=np.uint16)
    padded = so.pad_or_crop_scan(data)
    assert padded.shape[:2] == (128, 128)
    n = scan[0] * scan[1]
    sums, _ = ops.mean_dp_u64(torch.as_tensor(data, device=DEV), want_mean=False)
    fill, padded_sums = ops.pad_fill(sums, n, 128 * 128)
    np.testing.assert_array_equal(padded_sums.cpu().numpy().reshape(-1),
                                  padded.astype(np.int64).sum(axis=(0, 1)).reshape(-1))
    lin = torch.tensor([npix - 1, 0, 5], dtype=torch.int32, device=DEV)
    columns = ops.gather_bf_columns(torch.as_tensor(data, device=DEV), lin)
    top, left = (128 - scan[0]) // 2, (128 - scan[1]) // 2
    got = ops.pad_columns(columns, scan, fill, lin, 128, top, left)
    np.testing.assert_array_equal(got.cpu().numpy(),
                                  padded.reshape(128 * 128, npix)[:, lin.cpu().numpy()].T)


def test_a_scan_that_does_not_fit_is_refused():
    t = torch.zeros((1, 128), dtype=torch.uint16, device=DEV)
    lin = torch.zeros(1, dtype=torch.int32, device=DEV)
    with pytest.raises(_lib.QssbError):
        ops.pad_columns(t, (128, 1), t[0, :8], lin, 128, 1, 0)


def test_session_of_a_padded_scan_is_that_of_the_padded_block():
    counts = generate(CONFIGS["plain_32x32_det64"], device="cpu").counts.numpy()[:, :27]
    kw = dict(semiangle=20.0, scan_sampling=0.5, det_sampling=20.0 / 12.0, voltage_kV=300)
    a = B200SSBBackend(np.ascontiguousarray(counts), **kw)
    b = B200SSBBackend(so.pad_or_crop_scan(counts), **kw)
    assert a.scan_shape == (128, 128) and a.dc_value == b.dc_value
    np.testing.assert_array_equal(a.bf_inds_row, b.bf_inds_row)
    assert torch.equal(torch.view_as_real(a.G_qk), torch.view_as_real(b.G_qk))
