"""The attention backward (head_dim 64) hands registers from one warpgroup to another, and the wait for them has no limit: a build
with too few must be refused before a launch. Host arithmetic of the built library, no GPU."""

import ctypes

import pytest

from nanonemo_b200.csrc import build


@pytest.fixture(scope="module")
def library():
    if not build.LIB.exists():
        pytest.skip("kernel library not built")
    lib = ctypes.CDLL(str(build.LIB))
    lib.nnb_last_error.restype = ctypes.c_char_p
    return lib


@pytest.mark.parametrize("registers,fits", [(168, True), (128, True), (127, False), (120, False), (96, False)])
def test_a_build_whose_registers_do_not_add_up_is_refused(library, registers, fits):
    assert (library.nnb_flash_bwd_registers(registers) == 0) == fits
    if not fits:
        assert f"{registers} registers".encode() in library.nnb_last_error()


def test_the_launcher_asks_before_its_first_launch():
    text = (build.HERE / "flash_bwd.cu").read_text()
    launcher = text[text.index('extern "C" int nnb_flash_bwd('):]
    assert launcher.index("configure_bwd<false>()") < launcher.index("flash_bwd_kernel<false><<<")
    assert launcher.index("configure_bwd<true>()") < launcher.index("flash_bwd_kernel<true><<<")
    configure = text[text.index("static int configure_bwd()"):text.index('extern "C" int nnb_flash_bwd(')]
    assert "nnb_flash_bwd_registers(a.numRegs)" in configure
