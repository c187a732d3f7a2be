"""Host-side checks that need no GPU: the library loads, exports what the header declares, and
fails loudly (never falls back) when no device is present."""
import ctypes
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def declared_symbols(header: Path):
    text = header.read_text()
    return sorted(set(re.findall(r"W8A8_API\s+[\w\s\*]+?\b(w8a8_\w+)\s*\(", text)))


def test_header_symbols_are_exported(pkg):
    lib = pkg.load_library()
    names = declared_symbols(ROOT / "include" / "w8a8.h")
    assert len(names) >= 16
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/w8a8.h but not exported"
    from fish_audio_cpp_b200 import capi

    assert set(capi.EXPORTS) <= set(names)
    host = declared_symbols(ROOT / "include" / "w8a8_container.h")
    assert len(host) == 8 and set(capi.CONTAINER_EXPORTS) == set(host)
    for n in host:
        assert hasattr(lib, n), f"{n} declared in include/w8a8_container.h but not exported"


def test_shim_exports_reference_signatures(pkg):
    out = subprocess.run(["nm", "-D", "--defined-only", "-C", str(pkg.library_path())], capture_output=True,
                         text=True, check=True).stdout
    for sig in ["fish::kernels::int8_dequant_gemm_fp16(signed char const*, __half const*, int, __half const*, "
                "__half const*, __half const*, __half*, int, int, int, cublasContext*, CUstream_st*)",
                "fish::kernels::rms_norm(__half const*, __half const*, __half*, int, int, float, CUstream_st*)",
                "fish::kernels::silu_forward(__half*, int, CUstream_st*)",
                "fish::kernels::mul_forward(__half*, __half const*, int, CUstream_st*)",
                "fish::kernels::residual_add(__half*, __half const*, int, CUstream_st*)"]:
        assert sig in out, sig


def test_status_strings_and_workspace_arithmetic(pkg):
    lib = pkg.load_library()
    assert lib.w8a8_status_string(0) == b"ok"
    assert b"workspace" in lib.w8a8_status_string(5)
    # codes M*K (256-aligned) + scales M*G*4 (256-aligned)
    assert lib.w8a8_workspace_bytes(100, 64, 512, 64) == 51200 + 3328
    assert lib.w8a8_workspace_bytes(0, 64, 512, 64) == 0
    assert pkg.num_groups(2560, 256) == 10 and pkg.num_groups(2560, 0) == 1 and pkg.num_groups(100, 64) == 2


def test_no_silent_fallback_without_a_device(pkg):
    import torch

    if torch.cuda.is_available():
        pytest.skip("a device is present")
    with pytest.raises(pkg.W8A8Error) as e:
        pkg.Context(0, 1 << 20)
    assert e.value.status == 3  # W8A8_ERR_CUDA


def test_null_context_is_rejected(pkg):
    lib = pkg.load_library()
    assert lib.w8a8_linear(None, None, None, 64, None, None, None, None, 1, 8, 64, None, None) == 1
    assert b"context" in lib.w8a8_last_error()
    assert lib.w8a8_destroy(None) == 0


@pytest.mark.parametrize("n_kv", [1, 2, 8])
@pytest.mark.parametrize("batch", [1, 2, 3, 5, 8])
def test_one_launch_step_fills_the_gpu_whatever_the_tables_width(pkg, batch, n_kv):
    """The one-launch step's scratch, and with it the number of context slices, is the same for a short block table as for a long one."""
    from fish_audio_cpp_b200 import capi

    lib = pkg.load_library()
    d = capi.DecodeStack()
    d.n_layers, d.batch, d.dim, d.n_q_heads, d.n_kv_heads, d.head_dim, d.inter, d.group_size = 2, batch, 512, 4 * n_kv, n_kv, 128, 512, 64
    for f in ("layers", "final_norm", "rope_freqs", "positions", "seq_lens", "block_table", "k_cache", "v_cache", "x", "out"):
        setattr(d, f, 1 << 20)  # (never read: the answer is arithmetic)
    sizes = set()
    for blocks in (1, 17, 25, 26, 44, 128, 2048):
        d.max_blocks_per_seq = blocks
        sizes.add(lib.w8a8_decode_stack_workspace_bytes(ctypes.byref(d)))
    assert len(sizes) == 1 and sizes.pop() > 0


@pytest.mark.parametrize("n_kv", [1, 2, 4, 8])
def test_one_launch_scratch_for_a_batch_serves_smaller_ones(pkg, n_kv):
    from fish_audio_cpp_b200 import capi

    lib = pkg.load_library()
    d = capi.DecodeStack()
    d.n_layers, d.dim, d.n_q_heads, d.n_kv_heads, d.head_dim, d.inter, d.group_size, d.max_blocks_per_seq = 1, 256, 4 * n_kv, n_kv, 128, 256, 64, 64
    for f in ("layers", "final_norm", "rope_freqs", "positions", "seq_lens", "block_table", "k_cache", "v_cache", "x", "out"):
        setattr(d, f, 1 << 20)  # (never read: the answer is arithmetic)
    sizes = []
    for d.batch in range(1, 9):
        sizes.append(lib.w8a8_decode_stack_workspace_bytes(ctypes.byref(d)))
    assert sizes == sorted(sizes)


ROOM_148 = {2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 7: 15, 8: 15}  # what the occupancy query answers on 148 SMs


@pytest.mark.parametrize("sms,room", [(148, ROOM_148), (132, {2: 66, 3: 40, 4: 28, 6: 18, 8: 14}), (148, {})])
def test_attention_slices_run_at_once(pkg, sms, room):
    """More slices than one only where all their clusters run at once, for any batch, kv heads and table width; one for the shortest tables."""
    for n_kv in (1, 2, 4, 8):
        for batch in range(1, 33):
            for blocks in (0, 1, 8, 17, 25, 26, 36, 45, 60, 96, 128, 2048):
                s = pkg.debug_attention_slices(batch, n_kv, blocks, sms, room)
                assert s == 1 or batch * n_kv <= room.get(s, 0), (batch, n_kv, blocks, s)
                assert s == 1 or blocks > 8


@pytest.mark.parametrize("batch,n_kv,blocks,want", [(8, 8, 25, 1), (1, 8, 45, 3), (5, 8, 45, 3), (3, 8, 60, 4), (2, 8, 128, 6), (1, 8, 128, 8),
                                                    (12, 1, 128, 8), (8, 8, 128, 2), (10, 8, 128, 1), (1, 2, 25, 4)])
def test_attention_slices_that_were_measured_fastest(pkg, batch, n_kv, blocks, want):
    """Within 1 % of a decode layer of the fastest count."""
    assert pkg.debug_attention_slices(batch, n_kv, blocks, 148, ROOM_148) == want


@pytest.mark.parametrize("M,N,K,g,tiles", [
    (16, 2560, 9728, 64, 2), (16, 19456, 2560, 64, 2), (32, 2560, 9728, 64, 2), (16, 9728, 8704, 128, 2), (32, 155776, 2560, 256, 2),
    (16, 9728, 4096, 64, 2), (16, 9728, 22784, 256, 2), (29, 19456, 4096, 256, 2),
    (32, 2048, 16640, 64, 1), (16, 2290, 22784, 64, 1),   # no CTA has two tiles to share activations
    (32, 6144, 9728, 64, 1), (29, 6144, 14848, 64, 1), (20, 9728, 9728, 256, 1), (16, 9728, 9728, 64, 1),  # a lone third, fifth tile
    (19, 19456, 9728, 64, 1), (18, 19456, 2560, 128, 1),  # a lone ninth, more than 16 rows
    (16, 6144, 2560, 64, 1), (8, 2560, 9728, 64, 1), (12, 2560, 9728, 128, 1), (16, 2560, 9728, 256, 1)])
def test_decode_linear_takes_two_tiles_only_where_that_is_faster(pkg, M, N, K, g, tiles):
    """Packed and row-major weights alike, so that they give the same bits."""
    for kernel in (pkg.KERNEL_GEMV_PACKED, pkg.KERNEL_GEMV_TMA):
        form = pkg.debug_gemv_form(M, N, K, g, kernel=kernel)
        assert form[:2] == (8 if M <= 8 else 16 if M <= 16 else 32, tiles)


def test_decode_linear_form_refuses_what_the_kernels_refuse(pkg):
    assert pkg.debug_gemv_form(33, 2560, 2560, 64) is None and pkg.debug_gemv_form(8, 2560, 2432, 64) is None
    assert pkg.debug_gemv_form(8, 2560, 2560, 96) is None and pkg.debug_gemv_form(0, 2560, 2560, 64) is None


def test_gemm_form_follows_what_is_asked_for(pkg):
    """The rule that picks the tcgen05 GEMM's form, on the host: a width or split that is asked for is taken or refused, never
    replaced; one CTA per tile and pairs keep to their widths."""
    assert pkg.debug_gemm_form(8192, 19456, 2560, 256)[0] in (192, 256)
    assert pkg.debug_gemm_form(33, 2560, 9728, 64)[2] > 1, "few tiles and a long K: split"
    for g in (64, 128, 256):
        for bt in (32, 64, 96, 128):
            assert pkg.debug_gemm_form(150, 2560, 2560, g, token_width=bt, splits=1) == (bt, 1, 1)
            assert pkg.debug_gemm_form(150, 2560, 2560, g, token_width=bt, kernel=pkg.KERNEL_GEMM_PAIR) is None
            assert pkg.debug_gemm_form(33, 136, 1024, g, token_width=bt, splits=2) == (bt, 1, 2)
            # K = 1280 in groups of 256 is five groups: four runs of whole groups would leave the last one empty
            want = None if g == 256 else (bt, 1, 4)
            assert pkg.debug_gemm_form(97, 40, 1280, g, token_width=bt, splits=4) == want
        for bt in (192, 256):
            assert pkg.debug_gemm_form(150, 2560, 2560, g, token_width=bt) == (bt, 2, 1)
            assert pkg.debug_gemm_form(150, 2560, 2560, g, token_width=bt, splits=2) is None
    assert pkg.debug_gemm_form(8192, 2560, 9728, 64, splits=2) is None, "more tiles than the chip holds at once"
    assert pkg.debug_gemm_form(150, 2560, 2560, 256, token_width=100) is None
    assert pkg.debug_gemm_form(150, 2560, 2500, 250) is None
    # the widest form, where its register balance does not hold: another one takes the shape
    for g in (64, 128, 256):
        assert pkg.debug_gemm_form(256, 37888, 2560, g, kernel=pkg.KERNEL_GEMM_PAIR) == (256, 2, 1)
        assert pkg.debug_gemm_form(256, 37888, 2560, g, kernel=pkg.KERNEL_GEMM_PAIR, moved_registers=False) == (192, 2, 1)
        assert pkg.debug_gemm_form(8192, 19456, 2560, g, moved_registers=False) is not None


@pytest.mark.parametrize("M,N,K,g,want", [
    (2048, 2560, 9728, 256, (192, 2, 1)),  # 62 us; tiles of 96 tokens 74
    (150, 2560, 9728, 256, (64, 1, 2)),    # 12.9 us; tiles of 32, not split, 14.3
    (4001, 4097, 2560, 64, (192, 2, 1)),   # rows that leave element by element: 134 us; 256 wide 148
    (1441, 9728, 512, 128, (128, 1, 1)),  # a short K: 16.5 us; 32 wide 27.3
    (4438, 6144, 512, 256, (256, 2, 1)),  # 19.5 us; 96 wide 30.0
    (186, 19456, 3328, 256, (64, 1, 1)),  # a second wave of few tiles: 22.4 us; one wave of pairs of 192 25.0
    (64, 19456, 2560, 64, (32, 1, 1)),  # a wave that memory bounds: 17.0 us; 64 wide 18.3
])
def test_gemm_form_that_was_measured_fastest(pkg, M, N, K, g, want):
    assert pkg.debug_gemm_form(M, N, K, g) == want


def test_gemm_never_splits_the_hidden_width(pkg):
    """K = 2560: the sums of wqkv and w1|w3 are added in the order of the other kernels, whatever the number of tokens and rows."""
    for g in (64, 128, 256):
        for M in (33, 64, 97, 160, 300, 613, 2048, 8192):
            for N in (16, 96, 256, 1000, 2560, 4097, 6144, 19456):
                assert pkg.debug_gemm_form(M, N, 2560, g)[2] == 1


def test_product_never_touches_the_oracle():
    """Nothing under the package may import, link or read oracle/ (checker only)."""
    pat = re.compile(r"(^|\s)(import|from)\s+oracle\b|oracle/|w8a8o_|libw8a8_oracle|fishref")
    for p in list((ROOT / "fish-audio-cpp_b200").rglob("*")) + list((ROOT / "include").glob("*.h")):
        if p.suffix in {".py", ".cu", ".h", ".cuh"}:
            assert not pat.search(p.read_text()), p
