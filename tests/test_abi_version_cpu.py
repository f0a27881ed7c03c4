"""The bindings' structures are the header's: a shorter one would be read past its end."""
import ctypes
import os
import subprocess

from fluidml_b200 import cabi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_bindings_are_of_the_library(tmp_path):
    assert cabi.lib().fml_abi_version() == cabi.ABI_VERSION
    structures = {"fml_tensor": cabi.Tensor, "fml_gemm_params": cabi.GemmParams, "fml_conv_params": cabi.ConvParams, "fml_gemm_plan_info": cabi.GemmPlanInfo}
    source = tmp_path / "sizes.c"
    prints = "".join(f'printf("%zu ", sizeof({name}));' for name in structures)
    source.write_text(f'#include <stdio.h>\n#include "fluidml_cuda.h"\nint main(void) {{ {prints} printf("%d", FML_ABI_VERSION); return 0; }}\n')
    subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(source), "-o", str(tmp_path / "sizes")], check=True)
    sizes = [int(v) for v in subprocess.run([str(tmp_path / "sizes")], capture_output=True, text=True, check=True).stdout.split()]
    assert sizes == [ctypes.sizeof(s) for s in structures.values()] + [cabi.ABI_VERSION]
