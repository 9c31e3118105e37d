"""Collectives of one rank are copies: by a kernel where the buffers allow it, by the runtime where not."""
import os

import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("count", [1, 15, 16, 31, 32, 33, 8191, 8192, 8193, 8225, 8192 * 32 + 7,  # around a piece and a CTA of pieces
                                   148 * 8 * 256 * 4 * 16 - 32, 148 * 5 * 256 * 4 * 32 - 32, 148 * 5 * 256 * 4 * 32, 148 * 8 * 256 * 4 * 32 - 16, 148 * 8 * 256 * 4 * 32, 148 * 8 * 256 * 4 * 32 + 4097])  # of four pieces
@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (16, 0), (32, 64), (1, 0), (3, 8)])
def test_one_rank_copy(count, src_off, dst_off):
    os.environ.setdefault("UCCL_BOOTSTRAP_IFNAME", "lo")
    from unified_ccl_b200 import Communicator

    comm = Communicator(0, 1)
    src = torch.randint(0, 256, (count + 160,), device="cuda", dtype=torch.uint8)
    dst = torch.full((count + 160,), 77, device="cuda", dtype=torch.uint8)
    comm.allgather(src[src_off:src_off + count], dst[dst_off:dst_off + count])
    assert torch.equal(dst[dst_off:dst_off + count], src[src_off:src_off + count])
    assert (dst[:dst_off] == 77).all() and (dst[dst_off + count:] == 77).all()
    comm.destroy()


@gpu
def test_which_copy():
    """The kernel for aligned memory of this GPU; the runtime's copy for the rest and where CTAs are limited."""
    os.environ.setdefault("UCCL_BOOTSTRAP_IFNAME", "lo")
    from graph_util import KERNEL, MEMCPY, nodes
    from unified_ccl_b200 import Communicator, _C

    comm = Communicator(0, 1)
    x, y = torch.randn(4096, device="cuda"), torch.empty(4096, device="cuda")

    def kernel(call):
        call()
        (kind, name, _), = nodes(call)
        assert kind == MEMCPY or "local_copy_kernel" in name
        return kind == KERNEL

    assert kernel(lambda: comm.allgather(x, y))
    assert not kernel(lambda: comm.allgather(x[1:4000], y[:3999]))
    comm.set_blocks(4)
    assert not kernel(lambda: comm.allgather(x, y))
    comm.set_blocks(0)
    # pinned host memory, by address: copied as ever
    h = torch.arange(4096, dtype=torch.float32).pin_memory()
    assert not kernel(lambda: _C.allgather(comm.handle, h.data_ptr(), y.data_ptr(), 4096, 2, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(y.cpu(), h)
    comm.destroy()
