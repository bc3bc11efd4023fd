"""The one-rank copy on device buffers at every distance from a 16-byte boundary, at lengths around
the vector and CTA sizes: results are exact, and nothing around the destination is touched."""
import os

import pytest

torch = pytest.importorskip("torch")

from dccl_b200 import Communicator  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm(dccl_lib):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    saved = dict(os.environ)
    c = Communicator(rank=0, world=1, device=0)
    yield c
    c.finalize()
    os.environ.clear()
    os.environ.update(saved)


@pytest.mark.parametrize("nbytes", [1, 15, 16, 17, 31, 48, 63, 79, 200, 8191, 8192, 8193, 8192 + 63, 3 * 8192 + 31, 1 << 20])
def test_copy_at_every_pair_of_offsets(comm, nbytes):
    gen = torch.Generator(device="cuda").manual_seed(nbytes)
    src = torch.randint(0, 255, (nbytes + 32,), dtype=torch.uint8, device="cuda", generator=gen)
    offsets = (0, 1, 3, 4, 6, 8, 13, 15)
    for so in offsets:
        for do in offsets:
            dst = torch.full((nbytes + 32,), 0xAB, dtype=torch.uint8, device="cuda")
            comm.all_gather(src[so:so + nbytes], dst[do:do + nbytes])
            want = torch.full_like(dst, 0xAB)
            want[do:do + nbytes] = src[so:so + nbytes]
            assert torch.equal(dst, want), (nbytes, so, do)
