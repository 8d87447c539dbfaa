"""The cases of test_gpu_tile run the kernel they are there for: its
comparisons would also hold with the marching kernel on both sides."""

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import test_gpu_tile as T  # noqa: E402
from SWESimulators import BatchedEnsemble, _native  # noqa: E402


@pytest.mark.parametrize("case", T.CASES, ids=lambda c: "%dx%d-%s" % (c[0], c[1], c[3]))
def test_domains_run_the_tile_kernel(case):
    assert T._simulator(T.Common.CUDAContext(), case)._domain.kernel() == (_native.GO_KERNEL_TILE, 0)


@pytest.mark.parametrize("cases", T.BATCHES, ids=["quadratic", "linear-field"])
def test_batches_run_the_tile_kernel(cases):
    ctx = T.Common.CUDAContext()
    ens = BatchedEnsemble.BatchedCDKLM16([T._simulator(ctx, c) for c in cases])
    assert ens.batch.kernel() == (_native.GO_KERNEL_TILE, 0)
    assert ens.batch.tiles() == sum(-(-c[0] // 32) * -(-c[1] // 16) for c in cases)
