"""nanoRLHF-B200: a Blackwell-native RLHF training engine."""
__version__ = "0.1.0"
