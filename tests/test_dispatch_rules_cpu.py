"""Rules that pick a kernel variant, over all that they accept (no GPU needed)."""
import torch

from linear_moe_b200.ops import cuda as K


def test_scalar_decay_chunk_rule(monkeypatch):
    monkeypatch.setattr(K, "num_sms", lambda: 148)
    line = 8 * 128 * 148
    assert K._scalar_chunk(1, line, 1, 128) == K._scalar_chunk(4, -(-line // 16), 4, 128) == 128
    assert K._scalar_chunk(1, line - 1, 1, 128) == K._scalar_chunk(1, line, 1, 64) == 64
    for T in (1, 16, 64, 128, 192):                             # short sequences, however many heads
        assert K._scalar_chunk(256, T, 1000, 128) == 64
    assert K._scalar_chunk(256, 193, 1000, 128) == 128
    for chunk in (64, 128):                                     # every token in exactly one group, no group empty
        for BH in (1, 3, 16, 148, 1000):
            for T in list(range(1, 400)) + [4096, 16384, 100003]:
                G, cpg = K._scalar_groups(1, BH, T, chunk)
                assert cpg * 64 % chunk == 0 and (G - 1) * cpg * 64 < T <= G * cpg * 64


def test_tensor_map_views():
    """Views that tensor maps cannot describe (repeated rows, strided columns, odd strides) are copied, the others stay."""
    x = torch.zeros(2, 5, 3, 128, dtype=torch.bfloat16)
    wide = torch.zeros(2, 5, 3, 3 * 128, dtype=torch.bfloat16)
    for t in (x, wide[..., 128:256], x.transpose(1, 2).contiguous().transpose(1, 2), x[:, :, :1], x[:1], x[:, :1].expand(-1, 1, -1, -1)):
        assert K._tma_view(t) is t
    odd = torch.zeros(2, 5, 3, 129, dtype=torch.bfloat16)[..., :128]
    for t in (x[:, :, :1].expand(-1, -1, 3, -1), x[:1].expand(2, -1, -1, -1), x.transpose(2, 3), odd):
        c = K._tma_view(t)
        assert c.is_contiguous() and torch.equal(c, t)


def test_padded_tiles_own_their_rows():
    """A scan fetches a tile of C rows of n + 8 elements as one copy: every such row, the last one's end included, is in the tile's
    storage and in no other tile, and starts where 16-byte copies may."""
    for B, H, N, C, widths in ((1, 1, 1, 64, (128, 128, 128, 64)), (2, 3, 5, 64, (64, 64, 64, 64))):
        end = 0
        for t, n in zip(K._padded_tiles(B, H, N, C, widths, "cpu"), widths):
            assert t.shape == (B, H, N, C, n) and t.stride() == (H * N * C * (n + 8), N * C * (n + 8), C * (n + 8), n + 8, 1)
            assert t.storage_offset() >= end and t.storage_offset() % 8 == 0
            end = t.storage_offset() + B * H * N * C * (n + 8)
            assert end * t.element_size() <= t.untyped_storage().nbytes()


def test_views_that_start_off_a_boundary_are_copied():
    """16-byte copies and tensor maps need 16-byte aligned bases; a contiguous view of a larger buffer is contiguous wherever it starts."""
    n = 2 * 5 * 3 * 128
    for start in (1, 4, 7):
        t = torch.arange(n + start).bfloat16()[start:].view(2, 5, 3, 128)
        for f in (K._inner_contig, K._tma_view, K._aligned):
            c = f(t)
            assert c.data_ptr() % 16 == 0 and c.is_contiguous() and torch.equal(c, t)
    for t in (torch.zeros(2, 5, 3, 128), torch.zeros(n + 8).bfloat16()[8:].view(2, 5, 3, 128)):
        assert K._aligned(t) is t
