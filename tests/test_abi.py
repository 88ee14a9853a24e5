"""The C-ABI library builds, loads and exports exactly what include/mdb200.h
declares; the ctypes table agrees with the header.  No GPU calls."""
import ctypes
import os
import re

import pytest

from conftest import ROOT

HEADER = os.path.join(ROOT, "include", "mdb200.h")


def _declared():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    out = {}
    for m in re.finditer(r"\b(?:const\s+char\s*\*|int64_t|int)\s+(mdb_\w+)\s*\(([^;{]*?)\)\s*;", src, flags=re.S):
        args = m.group(2).strip()
        n = 0 if args in ("", "void") else len([a for a in args.split(",") if a.strip()])
        out[m.group(1)] = n
    return out


@pytest.fixture(scope="module")
def built():
    import __graft_entry__ as entry
    entry.build()
    import importlib
    return importlib.import_module("mineru-diffusion_b200")


def test_header_declares_the_path():
    decl = _declared()
    for name in ("mdb_kv_commit", "mdb_attn_block_paged", "mdb_attn_staircase_varlen", "mdb_gemm_bf16",
                 "mdb_gemm_splitk_partials", "mdb_gemm_gateup_swiglu", "mdb_add_rmsnorm", "mdb_qknorm_rope_commit",
                 "mdb_lmhead_sample", "mdb_unmask_decide", "mdb_last_device_status", "mdb_strerror"):
        assert name in decl


def test_library_exports_every_declared_symbol(built):
    handle = ctypes.CDLL(built._lib.LIB_PATH)
    for name in _declared():
        assert hasattr(handle, name), f"{name} declared in mdb200.h but not exported"


def test_ctypes_table_matches_header(built):
    decl = _declared()
    table = built._lib.SIGNATURES
    assert set(table) == set(decl)
    for name, n in decl.items():
        assert len(table[name][1]) == n, f"{name}: header has {n} parameters, ctypes table {len(table[name][1])}"


def test_host_side_checks_need_no_gpu(built):
    lib = built._lib.lib()
    assert lib.mdb_version() >= 100
    assert lib.mdb_strerror(0) == b"ok"
    assert b"aligned" in lib.mdb_strerror(-2)
    # argument validation happens before any launch
    assert lib.mdb_kv_commit(None, 8, None, 8, None, None, None, 4, 1024, 100, None) == -1
    assert lib.mdb_kv_commit(None, 8, None, 8, None, None, None, 0, 1024, 100, None) == 0    # empty input
    assert lib.mdb_attn_block_paged(None, None, None, None, None, 1, None, 2, 32, 16, 5, 10, 0.1, 1, None, 0, None) == -1
    assert lib.mdb_gemm_splitk_workspace_bytes(32, 4096, 2) == 2 * 32 * 4096 * 4
    assert lib.mdb_attn_paged_workspace_bytes(4, 32, 16, 1) == 0
    assert lib.mdb_attn_paged_workspace_bytes(4, 32, 16, 3) == 4 * 3 * 16 * 32 * 130 * 4
    assert lib.mdb_lmhead_workspace_bytes(32, 151936) > 0


def test_ops_refuse_cpu_tensors(built):
    import torch
    x = torch.zeros(4, 64, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        built.ops.linear(x, x)
    with pytest.raises(RuntimeError):
        built.ops.store_kvcache(x.view(4, 1, 64), x.view(4, 1, 64), x, x, torch.zeros(4, dtype=torch.int32))


def test_argument_blocks_match_the_header(tmp_path):
    """Size and field offsets of every struct of the header against its ctypes twin, as the C compiler sees them."""
    import importlib
    import subprocess
    lib = importlib.import_module("mineru-diffusion_b200._lib")
    names = re.findall(r"\}\s*(mdb_\w+)\s*;", open(HEADER).read())
    twins = {n: getattr(lib, "".join(p.capitalize() for p in n[len("mdb_"):].split("_"))) for n in names}
    assert len(twins) >= 10
    lines = [f'printf("{n} %zu\\n", sizeof({n}));' for n in twins]
    lines += [f'printf("{n}.{f} %zu\\n", offsetof({n}, {f}));' for n, t in twins.items() for f, _ in t._fields_]
    src = tmp_path / "sizes.c"
    src.write_text('#include <stddef.h>\n#include <stdio.h>\n#include "mdb200.h"\nint main(void) {\n' + "\n".join(lines) + "\nreturn 0; }\n")
    subprocess.run(["gcc", "-I", os.path.dirname(HEADER), "-o", str(tmp_path / "sizes"), str(src)], check=True)
    out = dict(l.split() for l in subprocess.run([str(tmp_path / "sizes")], capture_output=True, text=True, check=True).stdout.splitlines())
    for n, t in twins.items():
        assert int(out[n]) == ctypes.sizeof(t), n
        for f, _ in t._fields_:
            assert int(out[f"{n}.{f}"]) == getattr(t, f).offset, f"{n}.{f}"


# Callers built against an earlier header pass blocks of these sizes; a call reads no further.
BLOCK_BYTES = {"mdb_rows": 40, "mdb_gemm_args": 104, "mdb_residual_norm_args": 216, "mdb_rms_segment": 96, "mdb_gated_norm_args": 104,
               "mdb_part_norm_args": 104, "mdb_delta_prep_args": 376, "mdb_decay_args": 112, "mdb_mlstm_prep_args": 288, "mdb_decay_prep_args": 344,
               "mdb_scan_args": 304, "mdb_chunk_scan_args": 168, "mdb_moe_route_args": 88, "mdb_moe_plan_args": 56, "mdb_rotary_commit_args": 224,
               "mdb_window_attn_args": 200}


def test_argument_blocks_keep_their_size():
    import importlib
    lib = importlib.import_module("mineru-diffusion_b200._lib")
    for n, size in BLOCK_BYTES.items():
        assert ctypes.sizeof(getattr(lib, "".join(p.capitalize() for p in n[len("mdb_"):].split("_")))) == size, n


# A scan's block at the very end of a readable page.  The head count is past what a launch takes, so the call reads the whole block
# and is refused on the host.
SCAN_AT_PAGE_END = """
import ctypes as C, importlib, mmap, sys
sys.path.insert(0, {root!r})
lib = importlib.import_module("mineru-diffusion_b200._lib")
page = mmap.PAGESIZE
mem = mmap.mmap(-1, 2 * page)
base = C.addressof(C.c_char.from_buffer(mem))
libc = C.CDLL(None, use_errno=True)
assert libc.mprotect(C.c_void_p(base + page), C.c_size_t(page), 0) == 0
block = lib.ScanArgs()
block.mode, block.bs, block.heads, block.kv_heads, block.dim, block.dim_pad, block.vdim = 2, 1, 65536, 65536, 128, 128, 64
for name in ("q", "k", "v", "s0", "s1", "state", "cu_q", "start", "state_slot", "out"):
    setattr(block, name, 64)
at = base + page - {size}
C.memmove(at, C.addressof(block), {size})
handle = C.CDLL(lib.LIB_PATH)
handle.mdb_scan.argtypes = [C.c_void_p, C.c_void_p]
print(handle.mdb_scan(at, None), flush=True)
import os
os._exit(0)
"""


def test_a_scan_reads_no_further_than_its_block(built):
    import subprocess
    import sys
    code = SCAN_AT_PAGE_END.format(root=ROOT, size=BLOCK_BYTES["mdb_scan_args"])
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, (run.returncode, run.stderr[-400:])
    unsupported = int(re.search(r"MDB_ERR_UNSUPPORTED\s*=?\s*\(?(-?\d+)", open(HEADER).read()).group(1))
    assert int(run.stdout) == unsupported


def test_package_imports_without_the_private_stream_calls():
    """A torch built without CUDA has neither; the stream then comes from where it always may."""
    import subprocess
    import sys
    code = ("import importlib, torch\n"
            "for n in ('_cuda_getDevice', '_cuda_getCurrentRawStream'):\n"
            "    if hasattr(torch._C, n): delattr(torch._C, n)\n"
            "ops = importlib.import_module('mineru-diffusion_b200').ops\n"
            "torch.cuda.current_stream = lambda: type('S', (), {'cuda_stream': 17})()\n"
            "assert ops._stream() == 17\n")
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True, timeout=300)
