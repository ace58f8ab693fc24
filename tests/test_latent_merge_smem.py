"""Shared memory of the one-token latent merge for many sequences: a launch asks for what each of the kernel's two phases lays out."""
import pytest


@pytest.mark.parametrize("tt", [8, 16])
def test_room_for_both_phases(tt):
    from inference_engine_rust_b200.csrc import bindings as B
    for rank in range(8, 513, 8):
        asked = B.core().iert_latent_merge_wide_smem(tt, rank)
        assert asked >= 128 * (rank + 8) * 2 + 4 * tt * (rank + 4) + 4 * tt * 64        # weights, merged rows, weights of the runs
        assert asked >= 4 * 3 * tt * 128                                                # the sums of three quarters of the rank
