"""The bounds-checked build of the kernels (-DRMLX_BOUNDS): an index that leaves its table is
recorded (source file, line, index, limit) and the access is skipped or redirected to the reserved
page, so the launch returns normally. The library is chosen per process (RMLX_BOUNDS=1), hence the
child process. Stands in for a memory checker (the reference relies on Metal's validation layer and
its ``tracked_hazards`` feature, crates/rmlx-metal/src/device.rs:23-32)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r'''
import torch
from rmlx_b200 import _lib
from rmlx_b200.ops import decode as D
from rmlx_b200.ops.weights import LinearWeight

dev = torch.device("cuda:0")
hq, hkv, hd, K, page, max_blocks = 4, 2, 64, 256, 16, 4
g = torch.Generator(device=dev).manual_seed(0)
w = LinearWeight.random((hq + 2 * hkv) * hd, K, None, dev, generator=g)
x = torch.randn(1, K, device=dev, generator=g).to(torch.bfloat16)
norm = torch.ones(K, dtype=torch.bfloat16, device=dev)
kc = torch.zeros(8, hkv, page, hd, dtype=torch.bfloat16, device=dev)
vc = torch.zeros_like(kc)
bt = torch.tensor([[1, 2, 3, 4]], dtype=torch.int32, device=dev)
ang = torch.arange(256, device=dev, dtype=torch.float32)[:, None] * torch.arange(hd // 2, device=dev)[None, :] * 0.01
cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
q = torch.empty(1, hq, hd, dtype=torch.bfloat16, device=dev)
pos_ok = torch.tensor([5], dtype=torch.int32, device=dev)
pos_bad = torch.tensor([70], dtype=torch.int32, device=dev)      # block column 4 of a 4-column table

D.set_stream(True, ops="all")
assert _lib.cuda().rmlx_bounds_build() == 1
assert _lib.bounds_status() is None

def qkv(pos):
    D.rms_qkv_rope(x, w, norm, 1e-6, q, kc, vc, bt, pos, cos, sin, hq, hkv)
    torch.cuda.synchronize()

qkv(pos_ok)
assert _lib.bounds_status() is None and float(kc[1, :, 5].abs().sum()) > 0
kc.zero_(); vc.zero_()
qkv(pos_bad)
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "decode_stream.cu" and rec[2:] == (4, 4), rec
assert float(kc.abs().sum()) == 0 and float(vc.abs().sum()) == 0      # the append was skipped
assert _lib.bounds_status() is None                                   # reading clears the record
D.set_stream(False)
qkv(pos_bad)
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "decode_qkv_rope.cu" and rec[2:] == (4, 4), rec
assert float(kc.abs().sum()) == 0
D.set_stream(True, ops="all")

flat = torch.randn(1, (hq + 2 * hkv) * hd, device=dev, generator=g).to(torch.bfloat16)
D.rope_kv_write(flat, q, kc, vc, bt, pos_bad, cos, sin, hq, hkv)
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "rope_kv.cu" and rec[2:] == (4, 4), rec
assert float(kc.abs().sum()) == 0

# attention over 80 tokens with a 64-token table: the fifth page is read from the reserved page 0
lens = torch.tensor([80], dtype=torch.int32, device=dev)
out = D.flash_decode_paged(q, kc, vc, bt, lens)
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] in ("flash_decode.cu", "flash_decode_cluster.cu") and rec[2:] == (4, 4), rec
assert torch.isfinite(out.float()).all()

table = torch.randn(32, 64, device=dev, generator=g).to(torch.bfloat16)
D.embedding(table, torch.tensor([40], dtype=torch.int32, device=dev))
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "misc.cu" and rec[2:] == (40, 32), rec

# grouped products: an offset past the rows ends its expert early, a position past them has no row
from rmlx_b200.ops import narrow
from rmlx_b200.ops.quantized import pair_gemm
we = LinearWeight.random(256, 512, "q4", dev, experts=3, generator=g)
xe = torch.randn(6, 512, device=dev, generator=g).to(torch.bfloat16)
good = torch.tensor([0, 2, 3, 6], dtype=torch.int32, device=dev)
want = narrow.narrow_gemm(xe, we, offsets=good)
pairs = pair_gemm(xe, we, offsets=good)
torch.cuda.synchronize()
assert _lib.bounds_status() is None
out = torch.zeros_like(want)
narrow.narrow_gemm(xe, we, out=out, offsets=torch.tensor([0, 2, 3, 9], dtype=torch.int32, device=dev))
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "narrow_gemm.cu" and rec[3] == 7, rec
assert torch.equal(out[:3], want[:3]) and float(out[3:].abs().sum()) == 0
order = torch.tensor([0, 1, 6, 3, 4, 5], dtype=torch.int32, device=dev)
out.zero_()
narrow.narrow_gemm(xe, we, out=out, offsets=good, order=order, rows=6)
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "narrow_gemm.cu" and rec[2:] == (6, 6), rec
assert torch.equal(out[:2], want[:2]) and float(out[2].abs().sum()) == 0
out.zero_()
pair_gemm(xe, we, out=out, offsets=torch.tensor([0, 2, 3, 9], dtype=torch.int32, device=dev))
torch.cuda.synchronize()
rec = _lib.bounds_status()
assert rec is not None and rec[0] == "pair_gemm.cu" and rec[3] == 7, rec
assert torch.equal(out[:3], pairs[:3]) and float(out[3:].abs().sum()) == 0

# rows of W shorter than what is asked for ahead (one ring stage), and more row blocks than one: no address past the weight
for kind, k in (("q4", 512), ("q4", 1024), ("q8", 512), (None, 64)):
    for shares in (0, 1, 2):
        ws = LinearWeight.random(16 * 24 * 148 * 2 + 16, k, kind, dev, generator=g)
        narrow.narrow_gemm(torch.randn(3, k, device=dev, generator=g).to(torch.bfloat16), ws, shares=shares)
        torch.cuda.synchronize()
        rec = _lib.bounds_status()
        assert rec is None, (kind, k, shares, rec)

# and a clean call leaves no record
qkv(pos_ok)
assert _lib.bounds_status() is None
print("BOUNDS-OK")
'''


def test_bounds_checked_build_records_and_skips(dev):
    from rmlx_b200 import _build
    if not _build.CUDA_BOUNDS_LIB.exists():
        _build.build(kinds=("cuda_bounds",))
    env = dict(os.environ, RMLX_BOUNDS="1")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    proc = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=root, capture_output=True,
                          text=True, timeout=300)
    assert proc.returncode == 0 and "BOUNDS-OK" in proc.stdout, proc.stdout + proc.stderr


def test_normal_build_has_no_bounds_records(dev):
    from rmlx_b200 import _lib
    assert _lib.cuda().rmlx_bounds_build() == 0
    with pytest.raises(_lib.NativeError):
        _lib.bounds_status()
