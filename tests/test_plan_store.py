"""The plan names the visited store of the one-warp kernel as it is: 32-bit words
per warp, 1024 for n <= 16 as planned by default."""
import pytest

import sbfs

pytestmark = pytest.mark.gpu


def test_class_2_store_size():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    with sbfs.Engine() as eng:
        c = eng.plan()["classes"][2]
    assert c["kernel"] == "k_hash+k_mid" and c["slots"] == 1024
