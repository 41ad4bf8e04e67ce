"""Which tile width a product takes (host rule, no GPU needed)."""
import pytest

from kernel_align_b200 import _native


@pytest.mark.parametrize("m,n,k,tree,columns", [
    (512, 4096, 4096, 0, 128), (512, 4096, 16384, 0, 128), (2048, 1024, 512, 0, 128), (8, 8, 64, 0, 128),
    # the hidden gradient of an LM head: K is the vocabulary, the operand stream is all that counts
    (469, 4096, 128256, 0, 256), (1479, 1024, 128256, 0, 256), (206, 1024, 50304, 0, 256), (512, 4096, 16392, 0, 256),
    # slices summed in the kernel: the epilogue runs eight times
    (512, 4096, 28672, 1, 128), (128, 1024, 4096, 1, 128),
    # the narrow tiles would not fit the CTA pairs in one round
    (1024, 4096, 4096, 0, 256), (1024, 4096, 4096, 1, 256), (256, 37 * 256, 64, 0, 128), (256, 37 * 256 + 8, 64, 0, 256),
])
def test_narrow_tiles_where_they_pay(m, n, k, tree, columns):
    assert _native.cuda().ka_gemm_tile_columns(m, n, k, tree, 74) == columns
