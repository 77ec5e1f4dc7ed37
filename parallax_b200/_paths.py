"""Where the built library lives (shared by the build recipe and the loader)."""
import os
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
# PLX_SM100_LIBRARY points the loader at a libplx_sm100.so built elsewhere (same C ABI version)
LIB_PATH = os.environ.get("PLX_SM100_LIBRARY") or os.path.join(LIB_DIR, "libplx_sm100.so")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")


def host_path() -> str:
    """The C++ host side of eager calls.  It uses the C++ classes of the PyTorch and the Python it was compiled
    against, so their versions are in its name: after an upgrade there is none until it is built again."""
    import torch

    version = str(torch.__version__).replace("+", "_")
    return os.path.join(LIB_DIR, f"_plx_host.torch{version}.{sysconfig.get_config_var('SOABI')}.so")
