"""GEMM without communication: tiles split along K, activation in the epilogue, and the tensor-parallel layers of ranks that are all
in one process, against the fp32 product of the same bf16 operands, tile by tile."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
import cann_hccl_b200 as H  # noqa: E402
from cann_hccl_b200 import _lib as L  # noqa: E402
from cann_hccl_b200.parallel import fused_tp  # noqa: E402

pytestmark = pytest.mark.gpu
ACTS = {None: lambda t: t, "silu": torch.nn.functional.silu, "gelu": torch.nn.functional.gelu}


def operands(M, N, K, seed, n=1):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = [torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
    b = [(torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16) for _ in range(n)]
    return a, b


def check(c, ref):
    """Every 128 x 256 tile: bf16 rounding (2^-9 relative) of sums whose fp32 error is far below; activations do not amplify it
    (slopes below 1.2)."""
    M, N = ref.shape
    err = (c.float() - ref).abs().view(M // 128, 128, N // 256, 256).amax(dim=(1, 3))
    scale = ref.abs().view(M // 128, 128, N // 256, 256).amax(dim=(1, 3))
    bad = (err > scale * 2 ** -7).nonzero()
    assert bad.numel() == 0, "tiles off: %s" % bad[:8].tolist()


# one k step, then one row block split along K; few tiles, split and not; an odd number of row blocks; a last wave of a few tiles
# behind whole ones (pair, single); full waves exactly
SHAPES = [(128, 256, 64), (128, 256, 1088), (128, 256, 8192), (256, 256, 1088), (256, 256, 8192), (384, 768, 4096), (128, 8192, 3584), (128, 16384, 1024),
          (1024, 2048, 2112), (2560, 2048, 1024), (3200, 2048, 704), (2048, 2560, 64), (18944, 256, 256)]
# tiles of other widths than 256 columns: uneven column halves and a last tile of 64 (144 columns), several waves (192, last tile
# of 64; pair 224), a last tile of 176 of 208, single tiles of 128 and 80 columns split in four, pair tiles split in three and two,
# a last pair tile of 32 columns of 224
SHAPES += [(640, 4096, 2752), (640, 11008, 1024), (128, 28672, 1024), (384, 1280, 8192), (128, 2560, 8192), (256, 5120, 8192), (512, 3072, 4096),
           (1280, 5632, 1024), (2048, 8192, 1024)]
# pairs over an odd number of row blocks, the last half empty; just below the size from which they are used
SHAPES += [(2176, 1024, 512), (2176, 8192, 192), (1920, 2048, 512)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("act", [None, "silu", "gelu"])
def test_product(M, N, K, act):
    (a,), (b,) = operands(M, N, K, M + N + K)
    ref = ACTS[act](a.float() @ b.float().t())
    c = fused_tp.gemm(a, b, activation=act)
    check(c, ref)
    assert torch.equal(fused_tp.gemm(a, b, activation=act), c)


def test_silu_of_extreme_sums():
    """Sums that are the values themselves: bf16 rounding of the result (2^-9) on top of a few fp32 steps; exponentials beyond 2^126."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    x = torch.tensor([0., -1e-30, 1e-30, -1., 1., -20., 20., -86., -87., -87.5, -88., -88.5, -89., -100., 100., 3e38, -3e38], device="cuda")
    a = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16)
    a[:x.numel(), 0] = x.to(torch.bfloat16)
    b = torch.zeros(256, 64, device="cuda", dtype=torch.bfloat16)
    b[:, 0] = 1
    want = torch.nn.functional.silu(a[:, :1].float()).double().expand(128, 256)
    got = fused_tp.gemm(a, b, activation="silu").double()
    assert bool(((got - want).abs() <= want.abs() * 2 ** -8 + 2 ** -126).all()), got[:x.numel(), 0].tolist()


def test_output_aligned_to_16_bytes_only():
    (a,), (b,) = operands(256, 512, 512, 3)
    buf = torch.full((256 * 512 + 64,), 9.0, device="cuda", dtype=torch.bfloat16)
    out = buf[8:8 + 256 * 512].view(256, 512)
    fused_tp.gemm(a, b, out=out)
    check(out, a.float() @ b.float().t())
    assert bool((buf[:8] == 9).all()) and bool((buf[8 + 256 * 512:] == 9).all())


@pytest.mark.parametrize("p", [2, 3, 4])
@pytest.mark.parametrize("Ms,N,K", [(128, 256, 64), (256, 1024, 1152), (384, 512, 2048), (1152, 2048, 1024)])
def test_layers_of_local_ranks(p, Ms, N, K):
    xs, ws = operands(Ms, N, K, p + N, p)
    cfg = L.CommConfig.default()
    cfg.hcclBufferSize = 2
    c = H.Communicator.init_local(p, device=True, device_id=0, config=cfg)
    ys = fused_tp.all_gather_matmul(c, xs, ws, activation="silu")
    x = torch.cat([t.float() for t in xs])
    for r in range(p):
        check(ys[r], torch.nn.functional.silu(x @ ws[r].float().t()))
    hs, ws = operands(Ms * p, N, K, p + K, p)
    outs = fused_tp.matmul_reduce_scatter(c, hs, ws)
    assert c.sync() == 0, c.describe_status()
    full = sum(h.float() @ w.float().t() for h, w in zip(hs, ws))
    for r in range(p):
        check(outs[r], full[r * Ms:(r + 1) * Ms])
    c.destroy()


def test_communicating_kernels_on_virtual_ranks():
    """The kernels that communicators over several processes run, on virtual ranks (HCCL_TP_DIRECT=0): the whole fused-kernel file."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join(here, "test_gpu_fused_tp.py"), "-x", "-q", "-m", "gpu"],
                       env=dict(os.environ, HCCL_TP_DIRECT="0"), capture_output=True, text=True, cwd=os.path.dirname(here), timeout=1200)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1500:]
