"""A CTA that waits in vain for the sums of another one: the kernel ends, and the next GEMM is refused until the status has been read."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_reported(bmt_gpu):
    from bmtrain_b200.ops import _native
    from bmtrain_b200.ops import gemm as G

    lib = _native.cuda_lib()
    a = torch.randn(256, 128, device="cuda").half()
    want = G.gemm_nt(a, a)
    flag = torch.ones(1, dtype=torch.int32, device="cuda")
    _native.check(_native.entry("bmt_gemm_wait", "pp")(flag.data_ptr(), _native.stream()), "wait")
    torch.cuda.synchronize()
    assert int(flag) == 0 and torch.equal(G.gemm_nt(a, a), want)      # it was set: taken back, nothing to report
    _native.check(_native.entry("bmt_gemm_wait", "pp")(flag.data_ptr(), _native.stream()), "wait")
    torch.cuda.synchronize()                                          # ends after its two seconds
    with pytest.raises(RuntimeError, match="gave up waiting"):
        G.gemm_nt(a, a)
    assert lib.bmt_gemm_status() >> 16 == 12 and lib.bmt_gemm_status() == 0
    assert torch.equal(G.gemm_nt(a, a), want)
