"""The registered operator torch.ops.hashattn.decode_step as torch sees it, without a GPU: tracing, version counters,
a second copy of the package in one process."""
import os
import subprocess
import sys

import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx

from hashattention_b200 import torch_ops

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCALARS = (16, 16, 1.0 / 8, 0.1)


def step_args(device):
    """One sequence of two pages, one kv-head."""
    def make(*shape, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device=device)
    i32, f32 = torch.int32, torch.float32
    return dict(q=make(1, 4, 128), k_new=make(1, 1, 128), v_new=make(1, 1, 128), k_pages=make(2, 1, 256, 128),
                v_pages=make(2, 1, 256, 128), hash_pages=make(2, 1, 256, 4, dtype=i32), page_table=make(1, 2, dtype=i32),
                seq_lens=make(1, dtype=i32), wq=make(4, 36864), bq=make(4, 288, dtype=f32), wk=make(4, 36864),
                bk=make(4, 288, dtype=f32), q_codes=make(1, 4, dtype=i32), sel_idx=make(1, 4, 64, dtype=i32),
                sel_cnt=make(1, 4, dtype=i32), workspace=make(1 << 20, dtype=torch.uint8), status=make(1, dtype=i32),
                out=make(1, 4, 128))


def test_written_arguments_count_as_modified_in_place_on_fake_tensors_too():
    with FakeTensorMode():
        args = step_args("cuda")
        before = {n: t._version for n, t in args.items()}
        torch.ops.hashattn.decode_step(*args.values(), *SCALARS)
        changed = {n for n, t in args.items() if t._version != before[n]}
    assert changed == {"k_pages", "v_pages", "hash_pages", "q_codes", "sel_idx", "sel_cnt", "workspace", "status", "out"}


def test_operator_traces_to_one_node():
    with FakeTensorMode() as mode:
        args = step_args("cuda")
        graph = make_fx(lambda *a: torch.ops.hashattn.decode_step(*a, *SCALARS), tracing_mode="fake",
                        _allow_non_fake_inputs=True)(*args.values()).graph
    assert mode is not None
    calls = [n for n in graph.nodes if n.op == "call_function"]
    assert [n.target for n in calls] == [torch.ops.hashattn.decode_step.default] and len(calls[0].args) == 18 + len(SCALARS)


def test_operator_object_takes_further_registrations():
    for name in ("register_vmap", "register_autograd", "register_kernel", "register_fake"):
        assert callable(getattr(torch_ops.decode_step, name))


def test_package_loads_twice_in_one_process():
    """Its directory name is no identifier, so every program picks a module name of its own."""
    code = '''
import importlib.util, os, sys
root = os.path.join(sys.argv[1], "hashattention-1.0_b200")
for name in ("hashattention_b200", "another_name"):
    spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"), submodule_search_locations=[root])
    sys.modules[name] = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(sys.modules[name])
import torch
torch.ops.hashattn.decode_step.default
importlib.reload(sys.modules["another_name.torch_ops"])
torch.ops.hashattn.decode_step.default
'''
    subprocess.run([sys.executable, "-c", code, ROOT], check=True, timeout=300)
