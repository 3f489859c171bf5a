"""Where a call changes kernels: each path against the one beside it, at the sizes where a tile or a threshold ends."""

import pytest
import torch

import quashkv_b200 as qk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 3, 129, 6143, 6144, 6271, 9473])
def test_unpacked_codes_equal_the_packed_ones(n, dtype):
    """One byte per coordinate and packed rows, at every width, on both sides of the size from which the tensor-core
    kernel runs: whole numbers, so they are the same."""
    x = torch.randn(n, 128, generator=torch.Generator().manual_seed(n)).to(dtype).to(DEV)
    for bits in (1, 2, 3, 4):
        q = qk.MSEQuantizer(128, bits, seed=42, device=DEV)
        codes, norms = q.compress(x)
        packed, norms_p = q.compress_packed(x)
        assert torch.equal(qk.unpack_bits(packed, bits, 128), codes) and torch.equal(norms, norms_p)
    for bits in (2, 3, 4):
        q = qk.InnerProductQuantizer(128, bits, seed=42, device=DEV)
        codes, signs, norms = q.compress(x)
        packed, packed_s, norms_p = q.compress_packed(x)
        assert torch.equal(qk.unpack_bits(packed, bits - 1, 128), codes) and torch.equal(norms, norms_p)
        assert torch.equal(qk.unpack_bits(packed_s, 1, 128), signs)
