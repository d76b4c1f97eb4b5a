"""Registers of the GEMM's forms as ptxas reports them: 512 threads leave 128 each, and a main loop must not go through local memory
for what its epilogue warps keep."""
import importlib.util
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_form_spills_but_the_bf16_pair(tmp_path):
    spec = importlib.util.spec_from_file_location("nvfp4_build_script", os.path.join(ROOT, "nanogpt-120a_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    r = subprocess.run([build._nvcc(), *build.ARCH, *build.COMMON, "-Xptxas", "-v", "-c", os.path.join(build.CSRC, "gemm_tcgen05.cu"),
                        "-o", str(tmp_path / "gemm.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    forms = re.findall(r"Compiling entry function '(\S*nvfp4_gemm_tcgen05_kernel\S*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads"
                       r".*?Used (\d+) registers", r.stdout + r.stderr, re.S)
    assert len(forms) > 20
    spilling = {}
    for name, stores, loads, registers in forms:
        assert int(registers) <= 128
        if int(stores) or int(loads):
            # <rows, columns, element, store path, panel, pair, beside its predecessor>
            form = re.search(r"kernelILi(\d+)ELi(\d+)E(f|13__nv_bfloat16)L\S*?StorePathE(\d)ELi(\d)ELb([01])ELb([01])E", name).groups()
            spilling[form] = (int(stores), int(loads))
    # two CTAs on 128 x 256 bf16: no more than before one GEMM could run beside another
    pairs = [("128", "256", "13__nv_bfloat16", "1", "0", "1", beside) for beside in "01"]
    assert set(spilling) <= set(pairs), spilling
    assert all(stores <= 28 and loads <= 20 for stores, loads in spilling.values()), spilling
