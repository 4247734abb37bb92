"""Which kernel a product takes by its size (csrc/gemm/routes.h, skinny_gemm.cu): at sizes where both kernels were timed on one B200,
the faster one.  The rules are host code of the kernel library, which counts 148 SMs where there is no device."""
import pytest

from litevllm_b200 import ops
from litevllm_b200.ops import _lib


# (tokens, rows, K, us one tile per CTA, us persistent)
@pytest.mark.parametrize("T,N,K,one,many", [
    (129, 64, 2048, 7.3, 9.3), (129, 128, 4096, 10.8, 14.1), (512, 128, 4096, 11.6, 13.9), (1000, 64, 8192, 11.9, 22.1),
    (256, 256, 5632, 12.6, 17.2), (129, 512, 8192, 14.6, 22.8), (200, 1024, 8192, 19.2, 23.3), (512, 256, 12288, 17.3, 30.7),
    (768, 4096, 512, 11.2, 12.7), (1000, 4096, 1024, 14.9, 18.6), (640, 6144, 2048, 21.6, 24.9), (512, 8192, 2816, 28.1, 30.1),
    (300, 12288, 512, 12.2, 15.7),
    (129, 512, 512, 8.0, 6.7), (768, 128, 2048, 13.4, 9.8), (768, 128, 2816, 13.9, 11.3), (1000, 256, 2816, 14.2, 11.5), (300, 2048, 2048, 13.9, 10.8),
    (200, 2048, 5632, 24.0, 19.0), (600, 2048, 5632, 37.0, 22.0), (768, 2560, 2048, 18.6, 14.7), (512, 2560, 8192, 50.7, 29.3),
    (1000, 1024, 12288, 68.3, 33.5)])
def test_plain_products_of_129_to_1023_tokens(T, N, K, one, many):
    assert bool(_lib.kernels().fi_dense_gemm_persistent_pays(T, N, K)) == (many < one)
    assert ops._persistent_pays(T, N, K) == (many < one)


def test_from_1024_tokens_on_and_by_the_switch(monkeypatch):
    assert ops._persistent_pays(1024, 64, 8192)
    ops._persistent_pays.cache_clear()
    monkeypatch.setattr(ops, "_PERSISTENT_BY_SIZE", False)
    assert ops._persistent_pays(129, 64, 8192)
    ops._persistent_pays.cache_clear()
