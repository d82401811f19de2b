"""Which GEMM kernel a product without split K takes on 148 SMs (host rule, no GPU)."""
import pytest

from zero_to_hero_b200.ops import _lib

PAIRS = 2


# beside each the two times that decide, in us (one B200)
@pytest.mark.parametrize("M,N,K,kernel", [
    (16384, 3072, 768, PAIRS), (512, 384, 128, 64), (1024, 768, 768, 64), (2545, 1152, 384, 256), (200, 50264, 768, 256),
    (808, 4800, 1600, 256),     # one wave of single SMs 14.3, two of pairs 22.2
    (1920, 4800, 768, 256),     # two 16.5, three 19.9
    (2331, 9600, 768, 256),     # five 32.4, six 33.1
    (640, 50264, 768, PAIRS),   # seven 66.7, eight 58.8
    (2331, 50264, 768, PAIRS),  # 26 waves 211, 27 of pairs 176
    (1408, 50264, 512, PAIRS),  # 15 109, 16 104
    (1152, 50264, 192, 256),    # 12 71, 14 77: a short contraction is bound by its stores
])
def test_pairs_give_way_to_single_sms_only_where_they_lose(M, N, K, kernel):
    if not _lib.have_cuda_lib():
        pytest.skip("the kernel library is not built")
    assert _lib.cuda_lib().z2h_gemm_pick_kernel(M, N, K, 148) == kernel
