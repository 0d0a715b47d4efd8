"""The tiles' way on when a wait for the tensor cores runs out: builds of the library
in which it does, for every warp from its first product on, and for one lane of
the odd warps (which takes its warp along, beside warps that go on) from its
second product on, against the oracle word for word.  The waits themselves
complete in these builds, so nothing is left in flight."""
import os
import subprocess
import sys

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
GIVES_UP = {"all": "true", "odd": "(phase == 1 && threadIdx.x % 64 == 37)"}

pytestmark = pytest.mark.gpu


def check_all():
    """Runs in a process of its own, with the library of that build."""
    sys.path[:0] = [HERE, os.path.dirname(HERE)]
    import numpy as np

    import oracle_lib as O
    import test_gpu_batch
    import test_gpu_ntt_tiles
    import test_gpu_poseidon2_tiles
    import test_gpu_sky_tiles
    from provekit_b200.batch import Batch
    from provekit_b200.skyscraper import pow_solve

    ntt = test_gpu_ntt_tiles
    for kind in ("random", "edges", "top"):
        for shape in ((1, 1, 1), (8, 1, 2), (9, 3, 1), (11, 6, 4), (16, 1, 1), (17, 1, 8)):
            ntt.test_forward(*shape, kind)
    ntt.test_both_tile_sizes(20)
    ntt.test_encode(12, 5003, 60, 15)
    for log_n in (1, 9, 17):
        ntt.test_inverse_of_both_grids(log_n)
    sky = test_gpu_sky_tiles
    sky.test_hash_many(1, 544)
    sky.test_hash_many(129, 96)
    sky.test_compress_many((1 << 15) + 1)
    for encoding in (0, 1):
        sky.test_codeword_rows(encoding, 256, 8)
    for log_n in (1, 6, 8, 16):
        sky.test_subtrees(log_n)
    for n in (1, 129):
        test_gpu_poseidon2_tiles.test_permutation(n)
    test_gpu_poseidon2_tiles.test_hash(7)
    challenge, threshold = [1, 2, 3, 4], [0, 0, 0, 1 << 47]  # beyond the first, untiled batch
    exp = O.lib().pko_sky_pow_solve(O.p64(np.array(challenge, np.uint64)),
                                    O.p64(np.array(threshold, np.uint64)))
    assert exp >= 1 << 13
    assert pow_solve(challenge, threshold) == exp
    batch = Batch([4, 13, 10, 7, 11], seed=5)
    batch.run(use_graph=False)
    torch.cuda.synchronize()
    test_gpu_batch.check_batch(batch)  # its sumchecks against transcripts on the host


@pytest.mark.parametrize("warps", sorted(GIVES_UP))
def test_same_results(warps):
    from provekit_b200 import build
    lib = os.path.join(HERE, "_build", f"libprovekit_b200_alone_{warps}.so")
    os.makedirs(os.path.dirname(lib), exist_ok=True)
    build.build(lib=lib, defines=[f"-DPK_TILE_GIVES_UP={GIVES_UP[warps]}"])
    code = (f"import sys; sys.path[:0] = [{HERE!r}, {os.path.dirname(HERE)!r}]\n"
            f"from provekit_b200 import _lib\n_lib.LIB_PATH = {lib!r}\n"
            "import test_gpu_tile_alone as t\nt.check_all()\nprint('done')")
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                          timeout=600)
    assert done.returncode == 0 and "done" in done.stdout, done.stdout + done.stderr
