"""The FP64 form of the first draw's low product: floor of (l + 8 / 2^34) * A / 2^17, which the kernels get
from one multiply-add rounded to zero, is (l * A + 11) >> 17 for every 18-bit l, and everything added up
stays below 2^53 with an ulp of one."""


def test_every_low_part():
    a = 0x5DEECE66D
    for low in range(1 << 18):
        assert ((low << 34) + 8) * a >> 51 == (low * a + 11) >> 17
    magic = 3 << 51
    assert magic - 2 * a >= 1 << 52 and magic + (((1 << 18) * a + 12) >> 17) < 1 << 53
