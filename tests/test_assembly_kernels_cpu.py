"""Kernels of the assembly (colb_b200/csrc/assemble.cu) from their source on
the CPU, under the host emulation of the CUDA thread model (tests/simt/simt.h):
what the order of threads and blocks may not change."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _source(name):
    return open(os.path.join(ROOT, "colb_b200", "csrc", name)).read()


def _run(tmp_path, driver, inc, text):
    d = str(tmp_path)
    open(os.path.join(d, inc), "w").write(text)
    for f in ("simt.h", driver):
        shutil.copy(os.path.join(HERE, "simt", f), d)
    exe = os.path.join(d, "driver")
    subprocess.check_call(["g++", "-std=c++20", "-O1", "-pthread", os.path.join(d, driver), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_block_rows_by_a_block_and_by_a_cluster(tmp_path):
    src = _source("assemble.cu")
    text = src[src.index("struct BitRows {"):src.index("DV void set_bit(")]
    text += "constexpr int BR_CL = 8;\n" + src[src.index("struct BitHost {"):src.index("__global__ void k_diag_keys(")]
    # shared memory of each block of the cluster, not one for all
    text = text.replace("__shared__ int s_sum[32], s_of[BR_CL];", "int* s_sum = (int*)g_dyn_smem; int* s_of = s_sum + 32;")
    text = text.replace("__shared__ int s_total;", "int& s_total = s_of[BR_CL];")
    assert "__shared__" not in text
    _run(tmp_path, "bit_rows_test.cpp", "bit_rows.inc", text)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_contact_assembly_over_several_groups_of_a_warp(tmp_path):
    common, phys, eng = _source("common.cuh"), _source("physics.cuh"), _source("engine.cuh")
    text = common[common.index("struct d3 {"):common.index("HD double comp(")]
    text += "inline d3 ld3(const double* p) { return mk3(p[0], p[1], p[2]); }\n"
    text += phys[phys.index("DV void barrier3("):phys.index("// ---------------------------------------------------------- orthogonality")]
    text += eng[eng.index("DV int find_block("):eng.index("#define GS_LOOP")]
    text += _source("contact_hess.cuh").replace("#pragma once", "").replace('#include "common.cuh"', "")
    src = _source("assemble.cu")
    text += src[src.index("DV int stencil_np("):src.index("DV int other_vertex(")]
    text += src[src.index("constexpr int CA_PER = 8;"):src.index("// ---------------------------------------------------- block-Jacobi inverse")]
    for plain in ("double m[CA_PER][15], frame[CA_PER][9], w[CA_PER][12], gd[CA_PER], J[4][4];", "int v[CA_PER][4], type[CA_PER];"):
        kind, names = plain.split(" ", 1)
        assert plain in text
        text = text.replace(plain, f"Checked<{kind}> {names}")
    _run(tmp_path, "contact_assemble_test.cpp", "contact_assemble.inc", text)
