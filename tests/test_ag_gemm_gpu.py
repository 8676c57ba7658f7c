"""The GEMM whose input blocks arrive from peers, on one GPU: flags that are there already, and one that never comes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _call(flags, rank, world, rows, K, N, wait_ns, seed=0):
    from spark_engine_b200.ops import cuda as cu
    from spark_engine_b200.parallel import symm
    P, g = cu.P, torch.Generator(device=DEV).manual_seed(seed)
    a = torch.randn(world * rows, K, device=DEV, generator=g).bfloat16()
    b = torch.randn(N, K, device=DEV, generator=g).bfloat16()
    out = torch.full((world * rows, N), float("nan"), device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    f = torch.tensor(flags, dtype=torch.int32, device=DEV)
    rc = symm._lib().spark_gemm_bf16_ag(P(a), P(b), P(out), world * rows, N, K, K, N, 1, P(f), 7, rows, rank, world, wait_ns, P(status),
                                       cu.stream(), None)
    cu.check(rc, "spark_gemm_bf16_ag")
    torch.cuda.synchronize()
    return out, a.double() @ b.double().t(), status.tolist()


@pytest.mark.parametrize("rows,N", [(96, 128), (96, 384), (128, 640), (300, 256)])
@pytest.mark.parametrize("rank", [0, 2])
def test_blocks_that_have_arrived(rows, N, rank):
    """Flags at or past the sequence number; a rank's own flag is not looked at."""
    flags = [7, 8, 7]
    flags[rank] = 0
    out, ref, status = _call(flags, rank, 3, rows, 256, N, 10 ** 9)
    assert status[0] == 0
    assert ((out.double() - ref).norm() / ref.norm()).item() < 256 * 2.0 ** -23


def test_block_that_never_arrives():
    """The wait runs out, the status names the peer and what was expected and seen, and the kernel returns."""
    _, _, status = _call([0, 7, 6], 0, 3, 128, 128, 128, 10 ** 7)
    assert status == [5, 2, 7, 6]
