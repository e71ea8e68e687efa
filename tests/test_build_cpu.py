"""What the build checks of the compiled kernels. CPU."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
spec = importlib.util.spec_from_file_location("b2c_build", os.path.join(ROOT, "pydtnn_b200", "csrc", "build.py"))
build = importlib.util.module_from_spec(spec)
spec.loader.exec_module(build)


def _ptxas(mode, bsrc, stream, reskb, regs, both=0):
    name = f"_ZN3b2c14conv_tc_kernelILi{mode}ELi128ELi4ELb0ELi2ELi{bsrc}ELi{stream}ELb0ELi{reskb}ELb0ELb{both}EEEv14CUtensorMap_stS1_S1_S1_S1_NS_8TcParamsE"
    return (f"ptxas info    : Compiling entry function '{name}' for 'sm_100a'\nptxas info    : Function properties for {name}\n"
            f"    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads\nptxas info    : Used {regs} registers, used 1 barriers\n")


def test_kernels_whose_roles_share_registers_have_them_all():
    other = _ptxas(0, 0, 0, 0, 168) + _ptxas(0, 1, 2, 0, 126) + _ptxas(0, 2, 2, 4, 126) + _ptxas(0, 2, 0, 0, 168, both=1)        # no warps for the B tile
    assert build.check_role_registers(other) == 0
    assert build.check_role_registers(other + _ptxas(1, 0, 0, 0, 128) + _ptxas(0, 1, 0, 0, 128) + _ptxas(0, 2, 1, 0, 128)) == 3
    for few in (_ptxas(1, 0, 0, 0, 126), _ptxas(0, 2, 1, 0, 120)):
        with pytest.raises(RuntimeError, match="registers"):
            build.check_role_registers(other + few)


def test_the_check_knows_the_form_for_pairs_of_ctas():
    name = lambda text: text.replace("EEEv14CUtensorMap", "ELb1EEEv14CUtensorMap")            # its last template argument
    assert build.check_role_registers(name(_ptxas(0, 1, 0, 0, 128) + _ptxas(1, 0, 0, 0, 128))) == 2
    with pytest.raises(RuntimeError, match="registers"):
        build.check_role_registers(name(_ptxas(1, 0, 0, 0, 126)))
