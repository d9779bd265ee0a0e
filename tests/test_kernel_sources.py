"""Rules of the kernel sources that a run on the GPU shows only by hanging."""
from pathlib import Path

import multimesh_jax_b200

KERNELS = Path(multimesh_jax_b200.__file__).parent / "csrc" / "kernels"


def test_warps_reach_a_cluster_barrier_whole():
    """The aligned barrier instructions must be executed by a warp's lanes together; a loop or branch by lane ahead of
    them does not ensure that, so every one of them stands directly behind a warp barrier."""
    found = 0
    for path in sorted(KERNELS.glob("*.cu*")):
        lines = path.read_text().splitlines()
        for i, line in enumerate(lines):
            if "barrier.cluster." in line:
                found += 1
                assert lines[i - 1].strip() == "__syncwarp();", f"{path.name}:{i + 1}"
    assert found
