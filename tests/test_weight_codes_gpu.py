"""The weights that the tensor-core kernels multiply are, bit for bit, those of `dequant`: rows of the identity pick them out."""
import pytest
import torch

from llaminar_b200.gguf import GGMLType, quantize

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("qt", [GGMLType.Q4_K, GGMLType.Q5_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0, GGMLType.IQ3_S])
@pytest.mark.parametrize("rows", [32, 64, 128, 256])
def test_weights_are_those_of_dequant(qt, rows):
    """Scales of trained models, of zero, and (5 and 6 bits) too large for the short conversion, in one matrix."""
    from llaminar_b200 import ops
    n, k = 256, 768
    g = torch.Generator(device=DEV).manual_seed(rows)
    w = torch.randn(n, k, device=DEV, generator=g) * 0.05
    w[32:64] *= 30.0
    w[64:80, ::3] *= 100.0
    w[80:84] = 0.0
    if qt == GGMLType.Q4_K:
        w = w.clamp(-3, 3)                                  # larger ones are re-encoded when a model is loaded
    pw, sc = ops.pack_matrix(quantize(w, qt), qt, n, k), ops.scratch_for(DEV)
    want, eye, out = ops.dequant(pw).float(), torch.eye(k, device=DEV).bfloat16(), torch.empty(rows, n, device=DEV)
    for c in range(0, k, rows):
        ops.gemm(pw, eye[c:c + rows].contiguous(), out, scratch=sc)
        assert torch.equal(out, want[:, c:c + rows].T), c
