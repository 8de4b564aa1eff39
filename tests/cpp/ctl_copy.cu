// The copy of the control block that an emit hands to the host, against a fault that another
// CTA has stored in the host's block before, during or after it.
#include <cstdio>
#include <cstring>

#include "search.cuh"

using namespace pst;

int main()
{
	const uint32_t words = sizeof(BatchCtl) / 4;
	for (int emitting = 0; emitting < 2; emitting++) {
		for (uint32_t when = 0; when <= words; when++) {
			BatchCtl ctl, host;
			memset(&ctl, 0x5A, sizeof(ctl));
			memset(&host, 0, sizeof(host));
			ctl.fault = 0;  // the device's word is never set
			for (uint32_t t = 0; t < words; t++) {
				if (t == when)
					host.fault = 1;
				copy_ctl(&ctl, &host, t, words, emitting != 0);
			}
			if (when == words)
				host.fault = 1;
			if (emitting && host.fault != 1)
				return printf("a fault stored before word %u was lost\n", when), 1;
			host.fault = 0;
			if (memcmp(&ctl, &host, sizeof(ctl)) != 0)
				return printf("the other words differ\n"), 1;
		}
	}
	printf("ok\n");
	return 0;
}
