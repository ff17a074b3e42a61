"""Prompts that the tcgen05 attention kernel takes with two row tiles per CTA (test_kernel_choice.py holds them against the rule): heads that
share their keys in pairs; groups of one and of three heads, whose pairs are rows that follow one another, the last of them without a partner
or cut short."""

# q heads, kv heads, head size, (q rows, kv rows) of the packed sequences
PACKED = [
    (32, 8, 128, [(1500, 1500), (200, 300)]),
    (32, 4, 64, [(1500, 1500), (600, 640)]),
    (40, 40, 64, [(500, 600), (500, 500), (500, 500), (500, 530)]),
    (40, 40, 64, [(1410, 1410), (100, 140)]),
    (33, 11, 128, [(1500, 1600), (100, 100)]),
]
# q heads, kv heads, head size, position, rows over the cache
CACHED = [(32, 8, 128, 0, 1500), (32, 8, 128, 300, 1500), (32, 4, 64, 100, 1500), (40, 40, 64, 0, 1410), (40, 40, 64, 40, 1500), (33, 11, 128, 40, 1500)]
# heads, key heads, key size, value size, rows of a prompt
STACKS = [(40, 40, 64, 64, 1410), (32, 4, 64, 48, 1500), (33, 11, 128, 128, 1500)]
