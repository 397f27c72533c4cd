"""pyl_pk_bin of one field with its per-CTA partial sums in the workspace (reduced by
pk_part_reduce_kernel) against the same call adding to shared memory, where the
reduction's partition changes: fewer CTAs than a group of slices, one CTA per plane,
several, and the axis without k_per slots.

Tolerance: the same float32 values in chains of at most 2^16 additions either way; with
independent roundings a chain is off by 2^8 ulps of its sum, 256 * 2^-24."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 256 * 2.0 ** -24


@pytest.mark.parametrize('axis', [0, 1, 2])
@pytest.mark.parametrize('dims', [2, 3, 13, 16, 33, 96, 257])
def test_partial_sums_equal_shared_sums(dims, axis):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.Pk_library as PKL
    from pylians_gb300 import _lib
    from pylians_gb300._device import ptr, stream_ptr
    lib = _lib.load()
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    dk = torch.randn((dims, dims, dims // 2 + 1), dtype=torch.complex64, generator=g, device='cuda')
    full = lib.pyl_pk_workspace_size(dims, 1, axis)
    bare = lib.pyl_pk_workspace_size(dims, 2, 2) if axis == 2 else 0      # axis 2: the ring table
    mp, keep = PKL.ctypes_int_array([2])
    out = []
    for nbytes in (full, bare):
        s = torch.full((lib.pyl_pk_sums_len(dims, 1),), 7.0, dtype=torch.float64, device='cuda')
        ws = torch.full((max(nbytes, 1),), 255, dtype=torch.uint8, device='cuda')
        _lib.call('pyl_pk_bin', ptr(dk), None, 1, dk.numel(), dims, axis, mp, ptr(s),
                  ptr(ws) if nbytes else ctypes.c_void_p(None), nbytes, stream_ptr())
        out.append(PKL._split_sums(s.cpu().numpy(), dims, 1))
    for k in ('PH', 'P1', 'P2'):
        assert np.all(np.abs(out[0][k] - out[1][k]) <= TOL * out[1][k]), k
    assert np.all(np.abs(out[0]['P3'] - out[1]['P3']) <= TOL * out[1]['P3'][:, :1])
