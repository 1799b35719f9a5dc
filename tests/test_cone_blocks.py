"""CPU test of the plain march's corner blocks where the device has no room for them: the frame marches the texels
instead of failing."""
import json
import os
import subprocess

import pytest

from megamol_gb300 import build as nbuild

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_OF_MEMORY, LAUNCH_FAILURE = 2, 719  # cudaError_t


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fit") / "cone_blocks_fit")
    subprocess.run([nbuild.nvcc(), *nbuild.ARCH, *nbuild.NVCC_FLAGS, os.path.join(HERE, "cone_blocks_fit.cu"),
                    os.path.join(nbuild.CSRC, "cone_blocks.cu"), "-o", exe], check=True)
    return lambda limit, error: json.loads(subprocess.run([exe, str(limit), str(error)], check=True, capture_output=True,
                                                          text=True).stdout)


def test_no_room_for_the_blocks(fit):
    full = 1 + 65 ** 3 + 33 ** 3 + 17 ** 3  # block 0 and a block per texel corner of the levels
    have = fit(32 * full, OUT_OF_MEMORY)
    assert have == dict(have, error=0, nblocks=full, blocked=3, asked=[32 * full])
    none = fit(32 * full - 1, OUT_OF_MEMORY)
    assert none == dict(have, nblocks=1, blocked=0, asked=[32 * full, 32])  # the same walls
    assert fit(0, OUT_OF_MEMORY)["error"] == OUT_OF_MEMORY
    other = fit(0, LAUNCH_FAILURE)  # another error is the frame's
    assert other["error"] == LAUNCH_FAILURE and other["asked"] == [32 * full]
