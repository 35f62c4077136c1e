"""Builds tests/cpp/engine_main.cu, which reaches the engine's classes behind the C ABI."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def build_engine_program(directory):
    from molds_gb300 import build
    build.build()
    libdir = os.path.join(ROOT, "molds_gb300", "_build")
    exe = str(directory / "engine_main")
    subprocess.run([build.nvcc()] + build.ARCH + ["-std=c++17", "-O1", "-I", build.CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(HERE, "cpp", "engine_main.cu"), "-o", exe, "-L", libdir, "-lnddo_gb300",
                    "-Xlinker", f"-rpath={libdir}", "-lpthread"], check=True)
    return exe


def run_engine_program(exe, *args):
    return subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=300)


def write_molecule(directory, theory, mol):
    """theory: its number in the C ABI; mol: atomic numbers Z and xyz in bohr"""
    p = directory / "molecule.txt"
    p.write_text("\n".join([str(theory)] + [f"{int(z)} {x:.17g} {y:.17g} {w:.17g}" for z, (x, y, w) in
                                            zip(mol.Z, mol.xyz.reshape(-1, 3).tolist())]) + "\n")
    return str(p)
