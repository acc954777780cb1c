"""Where the native host path of short calls (csrc/fal_host.cpp) is built to and loaded from.

The extension reads the objects of the Python and the torch whose headers it was compiled with, field by field.  Its file
is named after both, so that a file left from before an upgrade is not found, rather than loaded wherever its
symbols still resolve.
"""
import os
import sys
import sysconfig

import torch


def host_path(lib_dir):
    python = sysconfig.get_config_var("SOABI") or sys.implementation.cache_tag
    return os.path.join(lib_dir, f"_fal_host.{python}.torch-{torch.__version__}-{(torch.version.git_version or '')[:12]}.so")
