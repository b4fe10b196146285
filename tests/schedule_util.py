"""The batched rasterisers' task shapes, chosen by a test: the forward takes an
item's measured cost from the workspace (the last array in it, one word per
tile) and walks the items whose cost is a good part of the total in 8x8 blocks."""
import torch

CONFIGS = [(8, 1), (8, 2), (16, 2), (16, 4), (16, 8), (32, 4), (32, 8)]  # tile size, pixels per lane
# words of the schedule (256 bytes after the flags): leading items walked in
# blocks; not 0 where the batch holds something odd
SCHED_HEAVY, SCHED_ODD = 76, 77


def item_cost(batch):
    L = batch.layout
    size = 4 * (int(L.num_items) + 1)
    return batch._ws(int(L.total_bytes) - (size + 255) // 256 * 256, int(L.num_items), torch.int32)


def _sched(batch, word):
    return int(batch._ws(int(batch.layout.off_flags) + 256, 80, torch.int32)[word])


def heavy_items(batch):
    return _sched(batch, SCHED_HEAVY)


def odd(batch):
    return _sched(batch, SCHED_ODD) != 0


def leaders(batch):
    """Items that lead a task (8x8 tiles: the left one of two in a superblock row)."""
    out = []
    for v, c in enumerate(batch.cameras):
        tw, th = (-(-c.width // batch.tile_size), -(-c.height // batch.tile_size))
        run = min(2, 1 << int(batch.layout.sb_log2[v])) if batch.tile_size == 8 else 1
        lead = torch.arange(tw) % run == 0
        out.append(lead.repeat(th))
    return torch.cat(out).to(batch.device)


def set_blocks(batch, mask):
    """The next forward walks the masked items in blocks and the others in
    whole tasks (up to some 600 masked items; none masked: no cost is set)."""
    item_cost(batch).copy_(torch.where(mask, -1, 1).to(torch.int32))


def masks(batch):
    """Two of them that walk every item in both shapes between them."""
    lead = leaders(batch)
    rank = torch.cumsum(lead.int(), 0)
    return [lead & (rank % 2 == k) if int(lead.sum()) > 1 else lead for k in (0, 1)]
