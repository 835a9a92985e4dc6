"""What the Makefile needs to know about Python and torch to build _torch_call.

  torch_flags.py id        one line that changes when the Python or the torch it is built for does
  torch_flags.py suffix    file name ending that only this Python imports (needs no torch)
  torch_flags.py cflags    compiler flags (headers, ABI, torch's version as a macro)
  torch_flags.py ldflags   library folders
"""
import importlib.metadata
import importlib.util
import sys
import sysconfig


def torch_id():
    spec = importlib.util.find_spec("torch")          # located, not imported: this runs on every make
    if spec is None:
        sys.exit("torch is not installed for " + sys.executable)
    return " ".join((sysconfig.get_paths()["include"], sys.version.split()[0], importlib.metadata.version("torch"), str(spec.origin)))


def suffix():
    return sysconfig.get_config_var("EXT_SUFFIX")


def cflags():
    import torch
    from torch.utils import cpp_extension
    folders = cpp_extension.include_paths() + [sysconfig.get_paths()["include"]]
    return " ".join(["-isystem " + folder for folder in folders] +
                    [f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
                     f"-DKM_TORCH_VERSION='\"{torch.__version__}\"'"])


def ldflags():
    from torch.utils import cpp_extension
    return " ".join("-L" + folder for folder in cpp_extension.library_paths())


if __name__ == "__main__":
    print({"id": torch_id, "suffix": suffix, "cflags": cflags, "ldflags": ldflags}[sys.argv[1]]())
