"""Arguments of small host functions, with stand-ins for CUDA."""
import types

import numpy as np
import pytest
import torch

from funlbm_b200 import _lib


class _Torch:
    """torch with two devices: streams 100 + index, current device 1."""
    device = torch.device

    class cuda:
        @staticmethod
        def current_device():
            return 1

        @staticmethod
        def current_stream(device=None):
            index = torch.device(device).index if isinstance(device, str) else device
            return types.SimpleNamespace(cuda_stream=100 + (1 if index is None else index))

    class _C:
        @staticmethod
        def _cuda_getCurrentRawStream(index):
            assert type(index) is int
            return 100 + index


@pytest.mark.parametrize("device,stream", [
    (None, 101), (torch.device("cuda"), 101), (torch.device("cuda", 0), 100),
    ("cuda", 101), ("cuda:0", 100), (0, 100),
])
def test_stream_of_any_device_argument(device, stream):
    assert _lib.stream_of(_Torch, device).value == stream


@pytest.mark.parametrize("pitch,pz", [
    (None, 34), (True, 40), (np.bool_(True), 40), (1, 40), (False, 33), (np.bool_(False), 33),
    (0, 33), (35, 35), (np.int64(48), 48),
])
def test_pitch_arguments(pitch, pz):
    from funlbm_b200.lattice import pitch_of

    got = pitch_of(pitch, (6, 5, 33), "fp16s")
    assert got == pz and type(got) is int
