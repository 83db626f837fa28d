"""CPU checks of the C ABI: the library builds, loads, and exports every symbol the header declares."""

import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def libpath():
    from glorcq_b200 import _build
    return _build.build()


def header_symbols():
    text = open(os.path.join(ROOT, "include", "glorcq_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(glq_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_exported(libpath):
    L = ctypes.CDLL(libpath)
    syms = header_symbols()
    assert len(syms) >= 15
    missing = [s for s in syms if not hasattr(L, s)]
    assert not missing, f"declared in include/glorcq_b200.h but not exported: {missing}"


def test_binding_covers_header(libpath):
    from glorcq_b200 import _lib
    assert set(header_symbols()) <= set(_lib.exported_symbols())


def test_status_strings_and_sizes(libpath):
    from glorcq_b200 import _lib
    L = _lib.lib()
    assert L.glq_version() >= 100
    for st in (0, -1, -2, -3, -4, -5):
        assert len(L.glq_status_string(st)) > 0
    # C1 expert projection 1408 x 2048, 2-bit: 44 tile pairs x 16 blocks x 2 tiles x (512 B codes + 64 B scales)
    assert L.glq_tiled_bytes(_lib.FMT_Q2, 1408, 2048, 1) == 44 * 16 * 2 * 576
    # the same fused with a second matrix of that shape (gate | up): twice the pairs
    assert L.glq_tiled_bytes(_lib.FMT_Q2, 1408, 2048, 2) == 88 * 16 * 2 * 576
    assert L.glq_tiled_bytes(_lib.FMT_Q4, 2048, 2048, 1) == 64 * 32 * 2 * 576
    assert L.glq_tiled_bytes(_lib.FMT_T2, 1408, 2048, 1) == 1408 * 2048 // 4
    assert L.glq_tiled_f16_bytes(64, 2048) == 64 * 2048 * 2
    assert L.glq_sv_bytes(1408, 64, 1) == 44 * 4096 == 1408 * 64 * 2
    # ragged shapes are padded to whole tile pairs and k blocks
    assert L.glq_tiled_bytes(_lib.FMT_T2, 17, 130, 1) == 1 * 2 * 2 * 512
    assert L.glq_rows_f32_count(17, 1) == 32


def test_host_side_argument_checks(libpath):
    """Errors decided on the host, before any launch: no GPU needed."""
    from glorcq_b200 import _lib
    L = _lib.lib()
    assert L.glq_turbo_dequant_matmul(None, None, None, None, None, 1, 8, 64, None) == -1
    assert L.glq_turbo_dequant_matmul(None, None, None, None, None, 0, 8, 64, None) == 0      # B == 0: no-op
    assert L.glq_turbo_dequant_matmul(None, None, None, None, None, -1, 8, 64, None) == -1
    assert L.glq_gptq_dequant_matmul(None, None, None, None, None, None, 0, 8, 64, 128, 1, 0, None) == 0
    assert L.glq_pack_gptq(None, None, None, 2, 16, 128, 128, None, 0, 1, None) == -1
    assert L.glq_grouped_matmul(None, None) == -1
    # expert-parallel phases: the peer-memory exchange needs its pointer tables, the other phases must not get them
    import ctypes as C
    d = _lib.MoeDesc()
    d.top_k, d.H, d.E = 2, 64, 4
    dummy = C.create_string_buffer(64)
    ptr = C.cast(dummy, C.c_void_p).value

    def ep_call(ep):
        return L.glq_moe_forward_ep(C.byref(d), ptr, 1, ptr, None, None, None, None, 0, None, 0, None, None, None, None,
                                    C.byref(ep))
    ep = _lib.MoeEp(0, 2, _lib.MOE_PHASE_EXCHANGE, 0, ptr, None, None)
    assert ep_call(ep) == -1                                   # no peers
    peers = _lib.EpPeers(ptr, ptr, ptr, ptr, 0)
    ep.peers = C.pointer(peers)
    assert ep_call(ep) == -1                                   # buffers too small for the step (half_elems 0)
    ep.phase = _lib.MOE_PHASE_EXPERTS
    assert ep_call(ep) == -1                                   # the staging buffer is not exchanged
    assert ep_call(_lib.MoeEp(2, 2, _lib.MOE_PHASE_EXPERTS, 0, ptr, None, None)) == -1   # rank outside the world
    assert ep_call(_lib.MoeEp(0, 2, _lib.MOE_PHASE_ALL, 0, ptr, None, None)) == -1      # world > 1 needs phases


def test_no_fallback_without_gpu():
    """Without a CUDA device the product path must fail loudly, not compute on the CPU."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("GPU present")
    from tests import cases
    d = cases.make_linear(1, 32, 128, rank=16)
    with pytest.raises((RuntimeError, AssertionError)):
        cases.to_b200_linear(d, device="cpu")


def test_native_host_path_binds_and_refuses_cpu_tensors(libpath):
    import torch
    from glorcq_b200 import _lib
    nat = _lib.native()
    assert set(nat.names()) <= set(_lib.exported_symbols())
    w = _lib.Weight(None, None, None, None, None, None, 16, 128, 0, 0)
    layer = nat.layer(_lib.FMT_Q2, 128, bytes(w))
    with pytest.raises(RuntimeError, match="x must be a CUDA tensor"):
        nat.linear(layer, torch.zeros(1, 128, dtype=torch.float16), None, None, None)
    with pytest.raises(RuntimeError, match="x must be fp16"):
        nat.linear(layer, torch.zeros(1, 128), None, None, None)
    with pytest.raises(TypeError):
        nat.linear(layer)
    with pytest.raises(RuntimeError, match="x_rot must be a CUDA tensor"):
        nat.turbo_matmul(*[torch.zeros(1, 4, dtype=torch.float16)] * 4)


@pytest.mark.parametrize("shape", [(1, 64), (2, 4, 64), (64,), (2, 256), (4, 192), (2, 0)])
def test_native_linear_refuses_rows_of_another_width(libpath, shape):
    """Decided before any look at the device; (2, 4, 64) holds as many values as four rows of 128."""
    import torch
    from glorcq_b200 import _lib
    nat = _lib.native()
    layer = nat.layer(_lib.FMT_Q2, 128, bytes(_lib.Weight(None, None, None, None, None, None, 16, 128, 0, 0)))
    with pytest.raises(RuntimeError, match=f"rows of 128 values, got {shape[-1]}"):
        nat.linear(layer, torch.zeros(shape, dtype=torch.float16), None, None, None)
    with pytest.raises(RuntimeError, match="at least one dimension"):
        nat.linear(layer, torch.zeros((), dtype=torch.float16), None, None, None)


@pytest.mark.parametrize("shape", [(1, 4, 64), (2, 4, 192), (1, 2, 0)])
def test_native_moe_refuses_rows_of_another_width(libpath, shape):
    import ctypes as C
    import torch
    from glorcq_b200 import _lib
    d = _lib.MoeDesc()
    d.H, d.I, d.E, d.top_k = 128, 64, 4, 2
    nat = _lib.native()
    block = nat.block(C.addressof(d), 0, 0, 0, 0)
    with pytest.raises(RuntimeError, match=f"rows of 128 values, got {shape[-1]}"):
        nat.moe(block, torch.zeros(shape, dtype=torch.float16), None, None, None, None, None)
    with pytest.raises(RuntimeError, match="must be a CUDA tensor"):
        nat.moe(block, torch.zeros(1, 4, 128, dtype=torch.float16), None, None, None, None, None)


def test_moe_block_takes_three_dimensions_once_built_too(libpath):
    from types import SimpleNamespace
    import ctypes as C
    import torch
    from glorcq_b200 import _lib
    from glorcq_b200.moe_block import GraphCompatibleMoeBlock
    blk = GraphCompatibleMoeBlock(SimpleNamespace(num_experts=4, top_k=2, norm_topk_prob=False, gate=torch.nn.Identity(), experts=None))
    blk._desc, blk._built = _lib.MoeDesc(), True
    blk._desc.H, blk._desc.I, blk._desc.E, blk._desc.top_k = 128, 64, 4, 2
    blk._native = (_lib.native().block(C.addressof(blk._desc), 0, 0, 0, 0), False, (0, 0, 0))
    with pytest.raises(ValueError):
        blk(torch.zeros(4, 128, dtype=torch.float16))
    with pytest.raises(RuntimeError, match="CUDA"):
        blk(torch.zeros(1, 4, 128, dtype=torch.float16))


@pytest.mark.parametrize("K", [64, 192, 0])
def test_native_group_refuses_rows_of_another_width(libpath, K):
    import torch
    from glorcq_b200 import _lib
    nat = _lib.native()
    group = nat.group(_lib.FMT_Q2, 128, 3, 16, 128, 0, 0, 0)
    with pytest.raises(RuntimeError, match=f"rows of 128 values, got {K}"):
        nat.grouped_linear(group, torch.zeros(2, K, dtype=torch.float16))
    with pytest.raises(RuntimeError, match="fp16 CUDA rows"):
        nat.grouped_linear(group, torch.zeros(2, 128, dtype=torch.float16))


def test_workspace_of_products_with_few_columns(libpath):
    """The x.U products of a prompt re-tile nothing: no workspace, whatever x will be; wider products need theirs."""
    import ctypes as C
    from glorcq_b200 import _lib
    L = _lib.lib()
    m = _lib.MMArgs()
    m.fmt, m.n_problems, m.max_rows, m.rows_stride, m.N, m.K = _lib.FMT_F16, 1, 333, 333, 64, 4096
    assert L.glq_mm_workspace_bytes(C.byref(m)) == 0
    m.x, m.ldx = 2, 4097                        # not on 16-byte boundaries
    assert L.glq_mm_workspace_bytes(C.byref(m)) == 0
    m.N = 520
    assert L.glq_mm_workspace_bytes(C.byref(m)) >= 333 * 4096 * 2
    # a prompt through a block: the buffers of 512 x 4 entries (h, outputs, x.U: 19 MB; shared expert 9 MB) and one product's
    # re-tiled rows (at most 2048 + 61 x 256 rows of 2304 channels), not those of 60 experts with 512 rows each
    d = _lib.MoeDesc()
    d.H, d.I, d.E, d.top_k, d.rank, d.fmt, d.group_size, d.router_rows, d.dense0_rows = 2048, 1408, 60, 4, 64, _lib.FMT_Q2, 128, 61, 192
    d.I_shared = 5632
    assert L.glq_moe_workspace_bytes(C.byref(d), 512) < (19 + 9 + 81 + 10) << 20


def test_shared_memory_limits_are_set_in_one_place():
    """A limit that is set without being noted in the same step can be lowered under another thread's launch (glq_common.cuh,
    reserve_smem)."""
    csrc = os.path.join(ROOT, "glorcq_b200", "csrc")
    found = [f for f in sorted(os.listdir(csrc)) for _ in re.findall(r"MaxDynamicSharedMemorySize", open(os.path.join(csrc, f)).read())]
    assert found == ["glq_common.cuh"]


def test_native_descriptor_follows_the_weight(libpath):
    """The host path's copy of a descriptor is made anew with the descriptor, whoever asked for that first."""
    import torch
    from glorcq_b200 import _lib
    from glorcq_b200.tiled import TiledWeight
    w = TiledWeight(_lib.FMT_Q2, 16, 128, 128, 1, "cpu")
    w.set_bias(torch.zeros(16))
    first = w.native
    assert w.native is first
    w.set_bias(None)
    w.desc_bytes()
    assert w.native is not first


def test_group_keeps_what_its_tables_point_to(libpath):
    import weakref
    import torch
    from glorcq_b200 import _lib
    from glorcq_b200.tiled import GroupedLinear, TiledWeight
    w = TiledWeight(_lib.FMT_Q2, 16, 128, 128, 1, "cpu")
    w.set_bias(torch.zeros(16))
    bias = weakref.ref(w.bias)
    group = GroupedLinear([w], None)
    w.set_bias(None)
    assert bias() is not None
    del group


def test_block_keeps_what_its_tables_point_to(libpath):
    import weakref
    from types import SimpleNamespace
    import torch
    from glorcq_b200 import _lib
    from glorcq_b200.moe_block import GraphCompatibleMoeBlock
    from glorcq_b200.quantized_linear import GLoRCQLinear
    from glorcq_b200.tiled import TiledWeight

    def layer(N, K):
        lin = GLoRCQLinear(K, N)
        lin._tiled = TiledWeight(_lib.FMT_Q2, N, K, 128, 1, "cpu")
        return lin
    experts = [SimpleNamespace(gate_proj=layer(128, 256), up_proj=layer(128, 256), down_proj=layer(256, 128)) for _ in range(2)]
    down = experts[1].down_proj._tiled
    down.set_bias(torch.zeros(256))
    bias = weakref.ref(down.bias)
    blk = GraphCompatibleMoeBlock(SimpleNamespace(num_experts=2, top_k=1, norm_topk_prob=False, gate=None, experts=experts))
    blk._build(torch.device("cpu"))
    down.set_bias(None)
    assert bias() is not None
    del blk
