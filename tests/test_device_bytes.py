"""Device bytes of handles whose solve needs other work arrays (host side only): the
Gauss-Seidel ring of a large grid takes the place of PCG work arrays, so that a handle
stays near the plain step's of the same grid (its entries are 16 bytes in both
precisions: a fifth more beside FP32 fields), and FP32-form solves of an FP64 scene
bring their own MIC(0) operands.
"""
import pytest


@pytest.mark.parametrize("side", [4096, 8192, 32768])
def test_gauss_seidel_beside_the_plain_step(side):
    import ifluids as ifl
    for precision, bound in ((ifl.FP64, 1.0), (ifl.FP32, 1.2)):
        assert ifl.device_bytes(ifl.GS, side, side, precision) <= bound * ifl.device_bytes(ifl.PLAIN, side, side, precision)


def test_flip_with_fp32_solves():
    import ifluids as ifl
    # fields and particles are FP64 either way; eight FP64 arrays of a solve against thirteen FP32 ones
    assert ifl.device_bytes(ifl.FLIP, 1024, 1024, ifl.FP32) <= ifl.device_bytes(ifl.FLIP, 1024, 1024, ifl.FP64)
